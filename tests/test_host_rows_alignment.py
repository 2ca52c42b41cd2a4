"""Rows whose address is no multiple of a value's size (a view into a byte buffer, which NumPy hands on as it is): they are
copied for the device, a kernel reads only aligned ones where they lie. A row's output does not depend on where it
was read from, so the results are those of an aligned copy to the bit."""
import os
import subprocess

import numpy as np
import pytest

import mlp_oracle as mo
from conftest import PKG

PROGRAM = r"""
#include "host_rows.hpp"
int main()
{
    alignas(16) char b[64];
    for (int o = 0; o < 32; o++)
        for (int reaches = 0; reaches < 2; reaches++)
            for (int host = 0; host < 2; host++)
                if (gbt::rows_in_place(b + o, reaches, host) != (reaches && host && o % 4 == 0)) return 1;
    return 0;
}
"""


def test_only_aligned_rows_are_read_in_place(tmp_path):
    (tmp_path / "rows.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(tmp_path / "rows.cpp"), "-o", str(tmp_path / "rows")],
                   check=True)
    assert subprocess.run([str(tmp_path / "rows")]).returncode == 0


def _at(x, offset):
    """x at an address `offset` bytes behind a multiple of 16"""
    b = np.zeros(x.nbytes + 32, dtype=np.uint8)
    first = -b.ctypes.data % 16 + offset
    y = b[first:first + x.nbytes].view(x.dtype).reshape(x.shape)
    y[...] = x
    assert y.ctypes.data % 16 == offset
    return y


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 6, 8, 15])
@pytest.mark.parametrize("rows", [1, 129, 40000])
def test_outputs_and_gradients(gpu_lib, rows, offset):
    rng = np.random.default_rng(rows)
    x = rng.uniform(-1.0, 1.0, size=(rows, mo.N_IN)).astype(np.float32)
    t = rng.normal(size=(rows, mo.N_USED)).astype(np.float32)
    with gpu_lib.WarmStart(seed=5) as w:
        want, (loss, grad) = w.forward(x), w.forward_backward(x, t)
        y, (l, g) = w.forward(_at(x, offset)), w.forward_backward(_at(x, offset), t)
    assert np.array_equal(y, want) and l == loss and np.array_equal(g, grad)
