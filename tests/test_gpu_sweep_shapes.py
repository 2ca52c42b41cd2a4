"""The FP64 sweeps' two tile shapes (narrow where the GPU has an SM for every tile, wide beyond that) form the same
terms in the same order: a solve alone and the same solve in a batch too large for narrow tiles have the same bits,
on meshes whose columns do not fill the tiles of either shape."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh,copies", [((6, 6, 9), 64), ((10, 8, 17), 20), ((12, 14, 10), 9)])
def test_narrow_and_wide_tiles_agree(mesh, copies, gpu_lib, meshgen, tmp_path):
    im, jm, km = mesh
    narrow = ((im - 1 + 1) // 2) * ((jm - 1 + 3) // 4)
    assert narrow <= 152 < narrow * copies
    meshgen.write_case(meshgen.annular_duct(IM=im, JM=jm, KM=km), str(tmp_path))

    def run(n):
        with gpu_lib.Solver([str(tmp_path)] * n, gpu_lib.FP64) as s:
            s.init_uniform()
            s.iterate(3, history=False)
            assert s.status().max() & 8 == 0
            return [s.get("cv", q) for q in (0, n - 1)]
    alone, batch = run(1), run(copies)
    assert np.array_equal(alone[0], batch[0], equal_nan=True) and np.array_equal(alone[0], batch[1], equal_nan=True)
