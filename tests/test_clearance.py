"""The clearance rule of static geometry (csrc/bfx_clearance.h, compiled with g++): a step fills its
halo beside the link kernel only while no solid cell lies within three cells of a lattice face.  A
restore applies it to the restored mask.  CPU only."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "numi-gpu-physics_b200", "csrc")


@pytest.fixture(scope="module")
def clear(tmp_path_factory):
    d = tmp_path_factory.mktemp("clearance")
    src, so = d / "c.cpp", d / "c.so"
    src.write_text('#include "bfx_clearance.h"\n'
                   'extern "C" int clear(const unsigned char* m, int nx, int ny, int nz, int part) {\n'
                   '    return bfx::solid_clear_of_faces(m, nx, ny, nz, (unsigned char)part);\n}\n')
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    f = ctypes.CDLL(str(so)).clear
    f.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 4
    return lambda m: bool(f(m.ctypes.data, m.shape[2], m.shape[1], m.shape[0], 0x3F))


@pytest.mark.parametrize("shape", [(9, 8, 11), (7, 7, 7), (6, 9, 9), (9, 4, 9), (9, 9, 5)])
def test_every_solid_cell_near_a_face_is_seen(clear, shape):
    mask = np.zeros(shape, np.uint8)
    mask[...] = 0x80  # a topology flag alone is not solid
    assert clear(mask)
    for cell in np.ndindex(shape):
        mask[cell] = 5
        assert clear(mask) == all(3 <= i < n - 3 for i, n in zip(cell, shape)), cell
        mask[cell] = 0x80
