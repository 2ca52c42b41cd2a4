"""The two forms of the sweeps' tiles in both precisions (FP32: a step's inputs read a step ahead on small grids; FP64:
narrow tiles there), for the mean flow and for the Spalart-Allmaras variable, form the same terms in the same
order: a solve alone and the same solve in a batch of more tiles than the GPU has SMs have the same bits. Meshes whose
columns do not fill the tiles, with odd and even numbers of steps (the last stage of the input ring holds one or
two)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 152
OPTIONS = {"mean flow": {}, "variable": {"turb": "200"}}


def _tiles(n, pa, pb):
    return ((n[0] - 2 + pa) // pa) * ((n[1] - 2 + pb) // pb)


@pytest.mark.parametrize("kind", list(OPTIONS))
@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("mesh", [(4, 4, 4), (6, 6, 9), (10, 8, 17), (12, 14, 10), (9, 18, 13)])
def test_forms_agree(kind, precision, mesh, gpu_lib, meshgen, tmp_path):
    im, jm, km = mesh
    one = _tiles(mesh, *((2, 4) if precision == "FP64" else (4, 8)))
    copies = SMS // one + 1
    assert one <= SMS < one * copies
    meshgen.write_case(meshgen.annular_duct(IM=im, JM=jm, KM=km, options=OPTIONS[kind]), str(tmp_path))
    names = ["cv", "dq"] + (["ev", "res_ev"] if kind == "variable" else [])

    def run(n):
        with gpu_lib.Solver([str(tmp_path)] * n, getattr(gpu_lib, precision)) as s:
            s.init_uniform()
            s.iterate(4, history=False)
            assert s.status().max() & 8 == 0
            return [[s.get(a, q) for a in names] for q in (0, n // 2, n - 1)]
    alone, batch = run(1)[0], run(copies)
    assert np.all(np.isfinite(alone[0][1:-1, 1:-1, 1:-1]))
    for got in batch:
        for name, a, b in zip(names, alone, got):
            assert np.array_equal(a, b, equal_nan=True), name
