"""The allocation-free sort's look-back words cover its blocks whatever its
entry limit: sorts of up to 256k entries run in quarter-size blocks, so a
smaller limit has more blocks per entry.  The sources are compiled (no GPU)
with other limits and the sizes compared at compile time."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
@pytest.mark.parametrize("limit", [1 << 10, 1 << 19, 1 << 20, 1 << 21])
def test_status_words_cover_the_blocks(tmp_path, limit):
    src = open(os.path.join(ROOT, "splat.js_b200/csrc/gs_static_sort.cu")).read()
    hdr = open(os.path.join(ROOT, "include/splat_b200.h")).read()
    hdr, k = re.subn(r"#define GS_STATIC_SORT_MAX .*", f"#define GS_STATIC_SORT_MAX ({limit}u)", hdr)
    assert k == 1
    src = src.replace("../../include/splat_b200.h", "splat_b200.h")
    # every sort of up to SS_MAX entries: the largest in full blocks and the largest in quarter blocks
    src += """
static_assert(gs::SS_STATUS >= 256ull * ((gs::SS_MAX + gs::SORT_BLOCK_ENTRIES - 1) / gs::SORT_BLOCK_ENTRIES), "");
constexpr uint32_t few = gs::SS_MAX < gs::RS_SMALL ? gs::SS_MAX : gs::RS_SMALL;
constexpr uint32_t quarter = gs::SORT_BLOCK_ENTRIES / 4;
static_assert(gs::SS_STATUS >= 256ull * ((few + quarter - 1) / quarter), "");
"""
    (tmp_path / "splat_b200.h").write_text(hdr)
    (tmp_path / "a.cu").write_text(src)
    r = subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(tmp_path), "-I",
                        os.path.join(ROOT, "splat.js_b200/csrc"), "-c", str(tmp_path / "a.cu"), "-o",
                        str(tmp_path / "a.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
