"""The sweeps on a block of more columns of tiles than 15 bits count (65540 nodes across the span, walls all round):
FP64, whose tiles are 2 columns wide there, against the mixed form's tiles of 4, at the tile tests' bound of 1e-5 for
increments rounded to FP32 (the CPU oracle, which agrees with FP64 to 1e-10, takes over a minute here)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_long_block(gpu_lib, meshgen, tmp_path):
    im, jm, km = 65540, 4, 4
    small = meshgen.annular_duct(IM=4, JM=jm, KM=km, bump=0.0, options={"turb": "0"})
    x = np.repeat(small.nodes[:1], im, axis=0)
    x[..., :2] *= (1.0 + np.linspace(0.0, 0.5, im))[:, None, None, None]
    patches = [meshgen.Patch("inlet", 5, (1, im - 1, 1, jm - 1, 1, 1)), meshgen.Patch("outlet", 6, (1, im - 1, 1, jm - 1, km, km))]
    for face, rng in ((1, (1, 1, 1, jm - 1, 1, km - 1)), (2, (im, im, 1, jm - 1, 1, km - 1)),
                      (3, (1, im - 1, 1, 1, 1, km - 1)), (4, (1, im - 1, jm, jm, 1, km - 1))):
        patches.append(meshgen.Patch("wall", face, rng))
    meshgen.write_case(dataclasses.replace(small, nodes=x, patches=patches), str(tmp_path))
    cv = {}
    for prec in (gpu_lib.FP64, gpu_lib.MIXED):
        with gpu_lib.Solver(str(tmp_path), prec) as s:
            assert tuple(s.dims()[:3]) == (im, jm, km)
            s.init_uniform()
            s.iterate(2, history=False)
            assert s.status()[0] & 9 == 0
            cv[prec] = s.get("cv")[1:-1, 1:-1, 1:-1]
    a, b = cv[gpu_lib.FP64], cv[gpu_lib.MIXED]
    assert np.all(np.isfinite(a)) and np.linalg.norm(a - b) < 1e-5 * np.linalg.norm(a)
