"""Wall faces on either side of the velocity count from which Cercignani-Lampis walls
run in a launch of their own (1089 and 1369 velocities; mixed: are redone by wider
CTAs), alone and in a table whose first solve is below it; with the flux pass redone,
too.  Against the oracle, with the tolerances of the fused path's other parity tests
(FP64 1e-11: exp / erfc / pow ulps and the order of sums; mixed 1e-5)."""
import pytest
import torch

import host
from conftest import fields_err, rel_err
from pyugks_b200 import configs
from pyugks_b200.fused import FusedSolver

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-11, "mixed": 1e-5}
DT_TOL = {"fp64": 1e-12, "mixed": 1e-5}


def channel(reflect, m, scheme="vanLeer"):
    return configs.channel(nblocks=1, n=4, nj=3, m=m, flux_method=scheme, reflect_type=reflect, alpha_n=0.5,
                           alpha_t=0.7, CFL=0.3)


def check(gpu, k, ora, tol):
    assert gpu.solve_state()[k]["status"] == 0
    assert fields_err(gpu.fields(k), ora.fields()) < tol
    assert rel_err(gpu.interior_f(k)[0], ora.interior_f()[0]) < tol
    b, ob = gpu.blocks[gpu.solve_block_ids(k)[0]], ora.blocks[0]
    assert rel_err(b.wall_cover[:4, 2].cpu().numpy(), ob.wall_cover[:4, 2]) < tol
    assert rel_err(b.wall_fluxes[:4, 2].cpu().numpy(), ob.wall_fluxes[:4, 2]) < tol


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("redo", [False, True])
@pytest.mark.parametrize("m", [32, 36])
@pytest.mark.parametrize("reflect", ["D", "S", "CL"])
def test_walls(cuda, reflect, m, redo, precision):
    case = channel(reflect, m)
    case["delta_dt"] = 0.05
    ora, gpu = host.OracleSim(case, "port"), FusedSolver(case, precision=precision)
    assert gpu.launches_per_step() == (7 if precision == "mixed" else 5 if reflect == "CL" and m == 36 else 4)
    ora.one_step()
    ora.one_step()
    gpu.step(2)
    if redo:  # dt grows by its limit, and each step's flux pass is redone
        ora.dt *= 0.5
        gpu.solves.view(torch.float64)[0] *= 0.5
    for _ in range(3):
        ora.one_step()
    gpu.step(3)
    st = gpu.solve_state()[0]
    assert st["retries"] == (3 if redo else 0)
    assert abs(st["dt"] - ora.dt) <= DT_TOL[precision] * ora.dt
    check(gpu, 0, ora, TOL[precision])


@pytest.mark.parametrize("precision,launches", [("fp64", 7), ("mixed", 9)])
def test_table_of_both(cuda, precision, launches):
    """Three segments; FP64: the walls' launch with them."""
    cases = [channel("CL", 16), channel("S", 36), channel("CL", 36, "WENO5")]
    gpu = FusedSolver(cases, precision=precision)
    assert gpu.launches_per_step() == launches
    gpu.step(3)
    for k, case in enumerate(cases):
        ora = host.OracleSim(case, "port")
        for _ in range(3):
            ora.one_step()
        check(gpu, k, ora, TOL[precision])
