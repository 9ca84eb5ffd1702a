"""The extent of the expert tiles' row copies, from the kernels' own header compiled for the host: no run reads past a buffer."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "tile_reads.h"
extern "C" int vecs(int left, int stage, int nb) { return qv::row_stage_vecs(left, stage, nb); }
"""


@pytest.fixture(scope="module")
def vecs(tmp_path_factory):
    d = tmp_path_factory.mktemp("tile_reads")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "qvb8_b200", "csrc"), "-o", str(d / "t.so"),
                    str(d / "t.cpp")], check=True)
    return ctypes.CDLL(str(d / "t.so")).vecs


@pytest.mark.parametrize("P", [128, 256, 384, 640, 768, 1408, 2048])
@pytest.mark.parametrize("nb", [3, 4, 5, 6, 7, 8])
def test_stages_of_a_row_end_with_the_row(vecs, P, nb):
    """a row's stages of 256 columns, back to back: each as long as its columns, the last no further than the row's last byte"""
    row_bytes, at = P * nb // 8, 0
    for st in range(-(-P // 256)):
        assert st * 32 * nb == at                                       # where the kernel's stage starts
        at += 16 * vecs(P - st * 256, 256, nb)
        assert at <= row_bytes
    assert at == row_bytes
