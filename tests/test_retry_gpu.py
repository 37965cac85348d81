"""The dt control of a fused step and the flux pass it redoes when the growth limit
changes dt: dt, time and the number of passes of every step, and the fields, against
the oracle.  Tolerances as in the fused path's other parity tests (FP64 1e-11, mixed
1e-5)."""
import numpy as np
import pytest
import torch

import host
from conftest import fields_err, rel_err
from pyugks_b200 import configs
from pyugks_b200.fused import FusedSolver

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-11, "mixed": 1e-5}
DT_TOL = {"fp64": 1e-12, "mixed": 1e-5}


def cut_dt(gpu, oras, which, factor):
    """dt of some solves cut: it grows back by the limit, a flux pass redone each step."""
    dt = gpu.solves.view(torch.float64).view(gpu.nsolves, -1)
    for k in which:
        dt[gpu.order[k], 0] *= factor
        oras[k].dt *= factor


def check(gpu, oras, precision):
    tol, dt_tol = TOL[precision], DT_TOL[precision]
    for k, ora in enumerate(oras):
        st = gpu.solve_state()[k]
        assert st["status"] == 0
        assert st["steps"] == ora.step and st["retries"] == ora.flux_passes - ora.step
        assert abs(st["dt"] - ora.dt) <= dt_tol * ora.dt
        assert abs(st["time"] - ora.time) <= dt_tol * ora.time
        assert fields_err(gpu.fields(k), ora.fields()) < tol
        for a, b in zip(gpu.interior_f(k), ora.interior_f()):
            assert rel_err(a, b) < tol


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scheme", ["vanLeer", "WENO5", "minmod"])
def test_dt_grows_back(cuda, scheme, precision):
    """Two blocks with an adsorbing wall (a redone pass moves its coverage again):
    five limited steps, then the limit no longer binds."""
    case = configs.channel(nblocks=2, n=6, nj=5, m=8, flux_method=scheme, reflect_type="S", CFL=0.3)
    case["delta_dt"] = 0.05
    ora, gpu = host.OracleSim(case, "port"), FusedSolver(case, precision=precision)
    for n in (2, 1, 1, 1, 1, 1, 3):
        for _ in range(n):
            ora.one_step()
        gpu.step(n)
        check(gpu, [ora], precision)
        if ora.step == 2:
            cut_dt(gpu, [ora], [0], 0.5)
    passes = ora.flux_passes - ora.step
    assert 0 < passes < 8  # some steps redone, the last ones not
    for bi, ob in zip(gpu.solve_block_ids(0), ora.blocks):
        assert rel_err(gpu.blocks[bi].wall_cover[:6, 2].cpu().numpy(), ob.wall_cover[:6, 2]) < TOL[precision]


def table(count):
    """Small solves of the three limiters in turn."""
    out = []
    for k in range(count):
        case = configs.cavity(n=3 + k % 4, nj=4, m=4 + 4 * (k % 2), vlim=4.0, Kn=0.1, CFL=0.3,
                              flux_method=("vanLeer", "WENO5", "minmod")[k % 3])
        case["delta_dt"] = 0.02
        out.append(case)
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("count,which", [(5, (1, 2)), (20, (0, 7, 19)), (20, range(20)), (130, (1, 64, 127, 128, 129))])
def test_some_solves_of_a_table(cuda, count, which, precision):
    """Lists of retrying solves over one and several groups of 32."""
    cases = table(count)
    oras, gpu = [host.OracleSim(c, "port") for c in cases], FusedSolver(cases, precision=precision)
    for cut in (False, True):
        if cut:
            cut_dt(gpu, oras, which, 0.5)
        for ora in oras:
            for _ in range(2):
                ora.one_step()
        gpu.step(2)
    retries = [st["retries"] for st in gpu.solve_state()]
    np.testing.assert_array_equal([r > 0 for r in retries], [k in which for k in range(count)])
    check(gpu, oras, precision)
