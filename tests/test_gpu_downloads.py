"""Downloads of fields from one handle by several host threads at a time: each call returns its own field."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [(9, 9, 17), (33, 33, 65)])
def test_several_threads(mesh, gpu_lib, meshgen, tmp_path):
    im, jm, km = mesh
    meshgen.write_case(meshgen.annular_duct(IM=im, JM=jm, KM=km), str(tmp_path))
    names = ["cv", "pv", "res", "faceK", "cell", "mut"]
    with gpu_lib.Solver(str(tmp_path), gpu_lib.MIXED) as s:
        s.init_uniform()
        s.iterate(3, history=False)
        want = {n: s.get(n) for n in names}
        wrong = []

        def work(n):
            for _ in range(30):
                if not np.array_equal(s.get(n), want[n], equal_nan=True):
                    wrong.append(n)
        pool = [threading.Thread(target=work, args=(n,)) for n in names]
        for t in pool:
            t.start()
        for t in pool:
            t.join()
    assert not wrong


# eddy viscosities of 1800, 65536 (the most that goes through device memory), 67584 and 1048576 values (one full pinned
# piece), conserved variables of five times as many (from one piece to five), downloaded from small to large, where
# the pinned memory grows, and from large to small
SIZES = [(9, 9, 17), (63, 31, 31), (63, 31, 32), (127, 127, 63)]


def test_sizes(gpu_lib, meshgen, tmp_path):
    dirs = []
    for q, (im, jm, km) in enumerate(SIZES):
        dirs.append(str(tmp_path / f"m{q}"))
        meshgen.write_case(meshgen.annular_duct(IM=im, JM=jm, KM=km), dirs[-1])
    rng = np.random.default_rng(2)
    want = [1.0 + 0.1 * rng.random((im - 1, jm - 1, km - 1, 5)) for im, jm, km in SIZES]
    for order in (1, -1):
        with gpu_lib.Solver(dirs, gpu_lib.FP64) as s:
            s.init_uniform()
            for q, a in enumerate(want):
                s.set_cv(a, q)
            for q in range(len(dirs))[::order]:
                mut, cv = s.get("mut", q), s.get("cv", q)
                assert np.array_equal(cv[1:-1, 1:-1, 1:-1], want[q])
                assert mut.size * 5 == cv.size and np.all(np.isfinite(mut))
