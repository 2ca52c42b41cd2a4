"""Restriction and prolongation that end in the receiving level's primitive variables and limiter (one launch each in a
driver's iteration) against the separate calls of the interface, on states whose corrected (and
restricted) cells the limiter has to repair: the same bits on both levels, the same status."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COARSE = 2


@pytest.mark.parametrize("precision,part,mach,seed,coarse", [("FP64", 0.04, 2.5, 1, False), ("FP64", 0.04, 2.5, 3, False),
                                                             ("FP64", 0.02, 3.0, 6, True), ("MIXED", 0.04, 2.5, 1, False),
                                                             ("MIXED", 0.04, 2.5, 3, False)])
def test_repairs_in_a_cycle(precision, part, mach, seed, coarse, gpu_lib, meshgen, tmp_path):
    """part of the cells, moved at up to mach in each direction; coarse: whether restricted cells need a repair too"""
    # (CFL 10 is the ramp's cap: the driver's begin of an iteration leaves it as it is)
    options = {"multigrid": "Y", "coarse_iter": str(COARSE), "CFL": "10.0", "turb": "0"}
    meshgen.write_case(meshgen.rotor_passage(IM=9, JM=9, KM=33, options=options), str(tmp_path))
    rng = np.random.default_rng(seed)
    state = []
    with gpu_lib.Solver(str(tmp_path), getattr(gpu_lib, precision)) as a, gpu_lib.Solver(str(tmp_path), getattr(gpu_lib, precision)) as b:
        for s in (a, b):
            s.init_uniform()
            s.iterate(COARSE + 1, history=False)
            if not state:
                q = s.get("cv")[1:-1, 1:-1, 1:-1].copy()
                u = rng.uniform(-mach, mach, size=q.shape[:3] + (3,))
                fast = rng.random(q.shape[:3]) < part
                q[fast, 1:4] = (q[..., :1] * u)[fast]
                q[fast, 4] = (2.5 + 0.5 * q[..., 0] * (u * u).sum(axis=-1))[fast]
                state.append(q)
            s.set_cv(state[0])
        a.solver_step()
        # source/Solver.cpp:91-112 call by call
        b.set_use_force(2, True)
        b.time_marching(1)
        b.res_calculate(1)
        b.resflux(1)
        b.restrict()
        b.primitive_vars(2)
        b.limit_vars(2)
        restricted = int(b.status()[0])
        b.time_marching(2)
        b.delta_cons()
        b.corner_treatment(2)
        b.interpolate(0)
        b.primitive_vars(1)
        b.limit_vars(1)
        corrected = int(b.status()[0])
        assert bool(restricted & 2) == coarse and corrected & 2
        assert int(a.status()[0]) == corrected
        for level in (1, 2):
            for name in ("cv", "pv"):
                assert np.array_equal(a.get(name, 0, level)[1:-1, 1:-1, 1:-1], b.get(name, 0, level)[1:-1, 1:-1, 1:-1], equal_nan=True), (name, level)
