"""FP64 wall faces on either side of the velocity count from which
Cercignani-Lampis walls run in a launch of their own (1089 and 1369 velocities),
alone and in a table whose first solve is below it; with the flux pass redone, too.  Against the oracle, with the
tolerance of the fused path's other parity tests (1e-11: exp / erfc / pow ulps and
the order of sums)."""
import pytest
import torch

import host
from conftest import fields_err, rel_err
from pyugks_b200 import configs
from pyugks_b200.fused import FusedSolver

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-11


def channel(reflect, m, scheme="vanLeer"):
    return configs.channel(nblocks=1, n=4, nj=3, m=m, flux_method=scheme, reflect_type=reflect, alpha_n=0.5,
                           alpha_t=0.7, CFL=0.3)


def check(gpu, k, ora):
    assert gpu.solve_state()[k]["status"] == 0
    assert fields_err(gpu.fields(k), ora.fields()) < FP64_TOL
    assert rel_err(gpu.interior_f(k)[0], ora.interior_f()[0]) < FP64_TOL
    b, ob = gpu.blocks[gpu.solve_block_ids(k)[0]], ora.blocks[0]
    assert rel_err(b.wall_cover[:4, 2].cpu().numpy(), ob.wall_cover[:4, 2]) < FP64_TOL
    assert rel_err(b.wall_fluxes[:4, 2].cpu().numpy(), ob.wall_fluxes[:4, 2]) < FP64_TOL


@pytest.mark.parametrize("redo", [False, True])
@pytest.mark.parametrize("m", [32, 36])
@pytest.mark.parametrize("reflect", ["D", "S", "CL"])
def test_walls(cuda, reflect, m, redo):
    case = channel(reflect, m)
    case["delta_dt"] = 0.05
    ora, gpu = host.OracleSim(case, "port"), FusedSolver(case)
    assert gpu.launches_per_step() == (5 if reflect == "CL" and m == 36 else 4)
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
    assert abs(st["dt"] - ora.dt) <= 1e-12 * ora.dt
    check(gpu, 0, ora)


def test_table_of_both(cuda):
    cases = [channel("CL", 16), channel("S", 36), channel("CL", 36, "WENO5")]
    gpu = FusedSolver(cases)
    assert gpu.launches_per_step() == 8  # three segments, two retry launches, the walls
    gpu.step(3)
    for k, case in enumerate(cases):
        ora = host.OracleSim(case, "port")
        for _ in range(3):
            ora.one_step()
        check(gpu, k, ora)
