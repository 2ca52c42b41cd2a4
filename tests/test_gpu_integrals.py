"""Inlet and outlet integrals against their formula (source/Ouput.cpp:9-107,282-300) in numpy, on states as they are and on
states with cells without a speed of sound or a total pressure (negative temperature, pressure, density), where what the
formula cannot form is not a number. 1e-12: sums of a few hundred terms in another order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAMMA = float(np.float32(1.4))                           # (the reference reads it in single precision)


def _section(pv, faces, k):
    p, q = pv[1:-1, 1:-1, k], pv[1:-1, 1:-1, k - 1]
    m = 0.5 * (p + q)
    s = faces[:, :, k - 1, :3]
    mc = m[..., 0] * (m[..., 1] * s[..., 0] + m[..., 2] * s[..., 1] + m[..., 3] * s[..., 2])
    return p, m, mc


def _expected(pv, faces, k_out, r):
    """(total-pressure ratio, efficiency) with r the nondimensional gas constant"""
    g, g1 = GAMMA, GAMMA - 1.0
    base, tt = [], []
    with np.errstate(all="ignore"):
        for k in (1, k_out):
            p, m, mc = _section(pv, faces, k)
            ma = np.sqrt(m[..., 1] ** 2 + m[..., 2] ** 2 + m[..., 3] ** 2) / np.sqrt(g * r * m[..., 5])
            fac = 1.0 + g1 / 2.0 * ma * ma
            pt = p[..., 4] * fac ** (g / g1)
            base.append(np.sum(pt ** (g1 / g) * mc) / np.sum(mc))
            tt.append(np.sum(p[..., 5] * fac * mc) / np.sum(mc))
        pr = base[1] ** (g / g1) / base[0] ** (g / g1)
        return pr, (pr ** (g1 / g) - 1.0) / (tt[1] / tt[0] - 1.0)


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("where", [None, "inlet", "outlet", "both"])
@pytest.mark.parametrize("what", ["energy", "density"])
def test_total_pressure_ratio_and_efficiency(precision, where, what, gpu_lib, meshgen, tmp_path):
    meshgen.write_case(meshgen.rotor_passage(IM=9, JM=9, KM=33), str(tmp_path))
    with gpu_lib.Solver(str(tmp_path), getattr(gpu_lib, precision)) as s:
        s.init_uniform()
        s.iterate(5, history=False)
        a = s.get("cv")[1:-1, 1:-1, 1:-1].copy()
        for k, name in ((0, "inlet"), (-1, "outlet")):
            if where in (name, "both"):
                a[3, 4, k, 4 if what == "energy" else 0] *= -5.0
        s.set_cv(a)
        pv, faces = s.get("pv"), s.get("faceK")
        got = np.asarray(s.integrals(1)).reshape(-1)
    cell = pv[5, 5, 5]
    r = cell[4] / (cell[0] * cell[5])
    pr, eff = _expected(pv, faces, pv.shape[2] - 1, r)
    tol = 1e-12 if precision == "FP64" else 1e-6          # (r comes from FP32 values in the mixed form)
    for a, b in ((got[2], pr), (got[3], eff)):
        assert np.isnan(a) == np.isnan(b), (got, pr, eff)
        assert np.isnan(a) or abs(a - b) <= tol * abs(b) * (1e3 if b is eff else 1.0), (got, pr, eff)
