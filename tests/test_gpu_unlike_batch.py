"""A batch of blocks that are long in different directions: the product of the batch's largest extents takes more than 32
bits, although no block does. Every solve equals the same solve alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MESHES = [(5, 5, 1400), (5, 1400, 5), (1400, 5, 5)]


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_blocks_long_in_different_directions(precision, gpu_lib, meshgen, tmp_path):
    a, b, c = (max(m[d] for m in MESHES) - 1 for d in range(3))
    assert a * b * c >= 2 ** 31
    dirs = []
    for q, (im, jm, km) in enumerate(MESHES):
        dirs.append(str(tmp_path / f"m{q}"))
        meshgen.write_case(meshgen.annular_duct(IM=im, JM=jm, KM=km, options={"turb": "0"}), dirs[-1])

    def run(d):
        with gpu_lib.Solver(d, getattr(gpu_lib, precision)) as s:
            s.init_uniform()
            h = s.iterate(2)
            return h, [s.get("cv", q) for q in range(len(d))]
    h, cv = run(dirs)
    for q, d in enumerate(dirs):
        h1, cv1 = run([d])
        assert np.all(np.isfinite(h[:, q, :2])) and np.array_equal(h[:, q], h1[:, 0], equal_nan=True)
        assert np.array_equal(cv[q], cv1[0], equal_nan=True)
