"""Ghost cells that belong to two patches: the fills then run one after another in the reference's order (inlets, outlets,
walls, interfaces and periodic pairs, mixing planes last), in place of side by side. The profile's number of launches of
the boundary stage tells which way a case runs. Against the CPU oracle, which fills in that order: 1e-11 normwise on the
ghosts after one evaluation (the same arithmetic on the same interior), the parity tests' 1e-10 on the field after
three iterations."""
import dataclasses

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

OPTIONS = {"turb": "0"}                                    # (k-face walls are not for Baldwin-Lomax)


def _boundary_launches(s):
    s.profile_begin()
    s.resflux(1)
    return s.profile_end()["boundary"][1]


def _ghost_layers(a):
    return [a[0, 1:-1, 1:-1], a[-1, 1:-1, 1:-1], a[1:-1, 0, 1:-1], a[1:-1, -1, 1:-1], a[1:-1, 1:-1, 0], a[1:-1, 1:-1, -1]]


def _small_inlets(meshgen, im, jm):
    # inlet patches of 2 x 2 cells
    return [meshgen.Patch("inlet", 5, (i, i + 1, j, j + 1, 1, 1)) for i in range(1, im - 1, 2) for j in range(1, jm - 1, 2)]


def _duct(meshgen, im, jm, km, extra, small_inlets=False):
    case = meshgen.annular_duct(IM=im, JM=jm, KM=km, options=OPTIONS)
    patches = list(case.patches)
    if small_inlets:
        patches = _small_inlets(meshgen, im, jm) + patches[1:]
    return dataclasses.replace(case, patches=patches + extra(meshgen, im, jm, km))


def _none(meshgen, im, jm, km):
    return []


def _wall_on_inlet(meshgen, im, jm, km):
    return [meshgen.Patch("wall", 5, (3, im - 2, 2, jm // 2, 1, 1))]


def _wall_on_periodic(meshgen, im, jm, km):
    return [meshgen.Patch("wall", 3, (2, im - 2, 1, 1, 2, km // 2))]


def _wall_on_tenth_inlet(meshgen, im, jm, km):
    # (its ghosts belong to that inlet patch alone; it is the case's 260th patch, 250 after the inlet)
    return [meshgen.Patch("wall", 5, _small_inlets(meshgen, im, jm)[9].rng)]


@pytest.mark.parametrize("extra,mesh,split,ordered", [(_none, (9, 9, 13), False, False), (_wall_on_inlet, (9, 9, 13), False, True),
                                                      (_wall_on_periodic, (9, 9, 13), False, True),
                                                      (_none, (33, 33, 7), True, False), (_wall_on_tenth_inlet, (33, 33, 7), True, True)])
def test_fills_in_order_where_patches_share_cells(extra, mesh, split, ordered, gpu_lib, oracle_mod, meshgen, tmp_path):
    meshgen.write_case(_duct(meshgen, *mesh, extra, split), str(tmp_path))
    o = oracle_mod.Oracle(str(tmp_path))
    with gpu_lib.Solver(str(tmp_path), gpu_lib.FP64) as s:
        s.init_uniform()
        s.iterate(3, history=False)
        o.run(3)
        inner = (slice(1, -1),) * 3
        assert rel_err(s.get("cv")[inner], o.get("cv")[inner]) < 1e-10
        o.set_cv(s.get("cv")[inner])                       # the same interior on both sides
        s.set_cv(o.get("cv")[inner])
        assert (_boundary_launches(s) == 5) == ordered
        o.resflux(1)
        for name in ("cv", "pv"):
            for a, b in zip(_ghost_layers(s.get(name)), _ghost_layers(o.get(name))):
                assert rel_err(a, b) < 1e-11, name


def test_mixing_plane_over_a_wall(gpu_lib, meshgen, tmp_path):
    """a wall on a mixing plane's face: the plane, filled last, sets the same ghosts as without the wall"""
    plain = meshgen.stage_passage(options=dict(OPTIONS))
    im, jm, km = plain.blocks[0].shape[:3]
    wall = meshgen.BlockPatch(meshgen.Patch("wall", 6, (2, im - 2, 2, jm - 2, km, km)), 1)
    shared = dataclasses.replace(plain, patches=plain.patches + [wall])
    got = []
    for name, case in (("plain", plain), ("shared", shared)):
        d = str(tmp_path / name)
        meshgen.write_multiblock_case(case, d)
        with gpu_lib.Solver(d, gpu_lib.FP64) as s:
            s.init_uniform()
            rng = np.random.default_rng(7)
            for slot in s.slots(0):
                a = s.get("cv", slot)[1:-1, 1:-1, 1:-1]
                s.set_cv(a * (1.0 + 1e-3 * rng.normal(size=a.shape)), slot)
            n = _boundary_launches(s)
            got.append((n, s.get("pv", s.slots(0)[0])[1:-1, 1:-1, -1], s.get("pv", s.slots(0)[1])[1:-1, 1:-1, 0]))
    assert got[0][0] < got[1][0]
    assert np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][2], got[1][2])


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("extra", [_none, _wall_on_inlet, _wall_on_periodic])
def test_variable_of_the_turbulence_model_in_order(extra, precision, gpu_lib, meshgen, tmp_path):
    """the Spalart-Allmaras variable's ghosts: the configured ratio on the inlet, zero on a wall that lies on it, and on a
    periodic face its partner's cells, also where a wall lies there"""
    im, jm, km = 9, 9, 13
    case = meshgen.annular_duct(IM=im, JM=jm, KM=km, options={"turb": "200", "ev_ratio": "3.0"})
    wall = extra(meshgen, im, jm, km)
    meshgen.write_case(dataclasses.replace(case, patches=list(case.patches) + wall), str(tmp_path))
    with gpu_lib.Solver(str(tmp_path), getattr(gpu_lib, precision)) as s:
        s.init_uniform()
        s.iterate(3, history=False)
        s.resflux(1)
        ev = s.get("ev").reshape(im + 1, jm + 1, km + 1)
    inlet = np.full((im + 1, jm + 1), 3.0)
    if extra is _wall_on_inlet:
        a, b, c, d = wall[0].rng[:4]
        inlet[a:b + 1, c:d + 1] = 0.0
    assert np.array_equal(ev[1:-1, 1:-1, 0], inlet[1:-1, 1:-1])
    assert np.array_equal(ev[1:-1, 1:-1, -1], ev[1:-1, 1:-1, -2])
    assert np.array_equal(ev[1:-1, 0, 1:-1], ev[1:-1, -2, 1:-1]) and np.array_equal(ev[1:-1, -1, 1:-1], ev[1:-1, 1, 1:-1])
    assert np.all(ev[0, 1:-1, 1:-1] == 0.0) and np.all(ev[-1, 1:-1, 1:-1] == 0.0)
