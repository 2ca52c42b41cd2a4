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
