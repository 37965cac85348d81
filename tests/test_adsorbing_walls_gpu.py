"""Several adsorbing walls on one block: their CTAs run side by side and share the
block's wall arrays.  Against the oracle, which treats them one after another, with
the tolerances of the fused path's other parity tests (FP64 1e-11: exp / erfc / pow
ulps and the order of sums; mixed 1e-5: FP32 storage of f and the fluxes)."""
import numpy as np
import pytest

import host
from conftest import fields_err, rel_err
from pyugks_b200 import configs
from pyugks_b200 import defs as D
from pyugks_b200.fused import FusedSolver

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-11, "mixed": 1e-5}
WALLS = (D.NORTH, D.SOUTH, D.WEST)


def box(models, n, nj, scheme):
    """A cavity with adsorbing north, south and west walls that re-emit by models."""
    case = configs.cavity(n=n, nj=nj, m=12, vlim=4.0, flux_method=scheme, Kn=0.1, CFL=0.3)
    for k, (face, model) in enumerate(zip(WALLS, models)):
        case["blocks"][0]["bc"][face] = configs.adsorbing(
            1.0 + 0.1 * k, gamma_f=0.3 + 0.2 * k, k_des=0.02, reflect_type=model, alpha_n=0.6, alpha_t=0.7,
            beta_n=0.2, beta_t=0.1)
    return case


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,nj,scheme", [(7, 10, "vanLeer"), (10, 7, "WENO5")])
@pytest.mark.parametrize("models", [("S", "CL", "D"), ("CL", "D", "S"), ("D", "S", "CL"), ("CL", "CL", "CL")])
def test_three_adsorbing_walls(cuda, models, n, nj, scheme, precision):
    case, steps, tol = box(models, n, nj, scheme), 10, TOL[precision]
    ora = host.OracleSim(case, "port")
    for _ in range(steps):
        ora.one_step()
    ob = ora.blocks[0]
    runs = []
    for _ in range(2):
        gpu = FusedSolver(case, precision=precision)
        gpu.step(steps)
        assert gpu.solve_state()[0]["status"] == 0
        b = gpu.blocks[0]
        runs.append([t.cpu().numpy() for t in (b.f, b.flux_macro_S, b.flux_macro_W, b.wall_cover, b.wall_fluxes,
                                               b.wall_dist)])
        assert fields_err(gpu.fields(), ora.fields()) < tol
        assert rel_err(gpu.interior_f()[0], ora.interior_f()[0]) < tol
        for face in WALLS:
            cells = n if face in (D.NORTH, D.SOUTH) else nj
            assert rel_err(b.wall_cover[:cells, face].cpu().numpy(), ob.wall_cover[:cells, face]) < tol
            assert rel_err(b.wall_fluxes[:cells, face].cpu().numpy(), ob.wall_fluxes[:cells, face]) < tol
        # the reflected distribution of the wall treated last stays in wall_dist (a
        # velocity along the wall has none: 0 / 0)
        got, want = b.wall_dist.cpu().numpy(), ob.wall_dist
        ok = np.isfinite(want)
        np.testing.assert_array_equal(np.isfinite(got), ok)
        assert rel_err(got[ok], want[ok]) < tol
    for x, y in zip(*runs):
        np.testing.assert_array_equal(x, y)
