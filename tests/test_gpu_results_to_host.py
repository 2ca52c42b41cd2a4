"""Results on their way to the host: fields larger than one piece of the download (1 M values) come back as they were
set, histories longer than the rows kept on the device (256) are those of shorter runs, and training in several
calls draws the minibatches of one call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [(9, 9, 17), (49, 65, 73)])
def test_field_round_trip(mesh, gpu_lib, meshgen, tmp_path):
    im, jm, km = mesh
    meshgen.write_case(meshgen.annular_duct(IM=im, JM=jm, KM=km), str(tmp_path))
    with gpu_lib.Solver(str(tmp_path), gpu_lib.FP64) as s:
        s.init_uniform()
        inner = (slice(1, -1),) * 3
        a = s.get("cv")[inner].copy()
        a *= 1.0 + 1e-3 * np.random.default_rng(im).normal(size=a.shape)
        s.set_cv(a)
        b = s.get("cv")[inner]
    assert np.array_equal(a, b)


@pytest.mark.parametrize("cycles", [256, 257, 600])
def test_history_in_one_run_and_in_two(cycles, gpu_lib, meshgen, tmp_path):
    meshgen.write_case(meshgen.annular_duct(IM=9, JM=9, KM=17), str(tmp_path))

    def run(parts):
        with gpu_lib.Solver([str(tmp_path)] * 2, gpu_lib.MIXED) as s:
            s.init_uniform()
            return np.concatenate([s.iterate(n) for n in parts])
    assert np.array_equal(run([cycles]), run([100, cycles - 100]), equal_nan=True)


@pytest.mark.parametrize("parts", [[5], [2, 3], [1, 1, 3]])
def test_training_in_parts(parts, gpu_lib, meshgen, tmp_path):
    meshgen.write_case(meshgen.annular_duct(IM=9, JM=9, KM=17), str(tmp_path))
    with gpu_lib.Solver(str(tmp_path), gpu_lib.MIXED) as s:
        s.init_uniform()
        s.iterate(5, history=False)
        got = []
        for p in ([5], parts):
            with gpu_lib.WarmStart(seed=3) as w:
                w.add_solves(s, [[1.2, 1.0, 0.0]])
                for n in p:
                    w.train(n, batch=640)
                    x = np.zeros((9000, 64), dtype=np.float32)
                    w.forward(x)                             # (more rows than a minibatch, between the calls)
                got.append(w.get_params())
    assert np.array_equal(got[0], got[1])
