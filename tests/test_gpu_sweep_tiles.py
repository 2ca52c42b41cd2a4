"""LU-SGS sweeps on meshes at the edges of their tiles (4 x 8 grid columns, marched along k through a ring of
six steps): columns that fill tiles exactly, that leave a remainder of one or all but one, a single
ragged tile, fewer steps than the ring holds and many more. FP64 against the CPU oracle after three
iterations, at the tolerances of the other parity tests (the GPU reassociates sums and contracts
multiply-adds: 1e-9 on the history, 1e-10 normwise on the field). The mixed form against the FP64 form:
each iteration rounds Q's increments to FP32 (6e-8), so three of them stay far below 1e-5."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

HIST_COLS = [0, 1, 6, 7, 8, 11]        # iter, Res.dens, m_in, m_out, PR, CFL (the duct's efficiency is 0 / 0)
MESHES = [(5, 9, 9), (4, 8, 7), (6, 10, 12), (9, 17, 9), (13, 11, 21), (5, 18, 40), (8, 9, 5)]


@pytest.mark.parametrize("mesh", MESHES)
def test_sweeps_on_ragged_tiles(mesh, gpu_lib, oracle_mod, meshgen, tmp_path):
    im, jm, km = mesh
    meshgen.write_case(meshgen.annular_duct(IM=im, JM=jm, KM=km), str(tmp_path))
    o = oracle_mod.Oracle(str(tmp_path))
    ref = o.run(3)
    inner = (slice(1, -1),) * 3
    with gpu_lib.Solver(str(tmp_path), gpu_lib.FP64) as s:
        s.init_uniform()
        h = s.iterate(3)[:, 0, :]
        cv, dq = s.get("cv")[inner], s.get("dq")
        assert s.status()[0] & 8 == 0
    a, b = h[:, HIST_COLS], ref[:, HIST_COLS]
    assert float(np.max(np.abs(a - b) / np.abs(b))) < 1e-9
    assert rel_err(cv, o.get("cv")[inner]) < 1e-10
    with gpu_lib.Solver(str(tmp_path), gpu_lib.MIXED) as s:
        s.init_uniform()
        s.iterate(3, history=False)
        assert s.status()[0] & 8 == 0
        mixed = s.get("cv")[inner]
        assert np.linalg.norm(mixed - cv) < 1e-5 * np.linalg.norm(cv)
        assert np.all(np.isfinite(s.get("dq"))) and np.all(np.isfinite(dq))


def test_sweeps_of_a_ragged_batch_equal_single_solves(gpu_lib, meshgen, tmp_path):
    dirs = []
    for q, (im, jm, km) in enumerate(MESHES):
        dirs.append(str(tmp_path / f"m{q}"))
        meshgen.write_case(meshgen.annular_duct(IM=im, JM=jm, KM=km), dirs[-1])
    for prec in (gpu_lib.FP64, gpu_lib.MIXED):
        with gpu_lib.Solver(dirs, prec) as s:
            s.init_uniform()
            s.iterate(3, history=False)
            together = [s.get("cv", q) for q in range(len(dirs))]
        for q, d in enumerate(dirs):
            with gpu_lib.Solver(d, prec) as s:
                s.init_uniform()
                s.iterate(3, history=False)
                assert np.array_equal(together[q], s.get("cv"))
