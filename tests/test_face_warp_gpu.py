"""The FP64 face pass (a face per warp) at the edges of its work: velocity
counts around the warp size, blocks that are no multiple of the strips its work
items are ordered in, a curvilinear grid, and velocity grids described without
their tensor structure.  Against the oracle, with the tolerance of the fused
path's other parity tests (1e-11: exp / erfc / pow ulps and the order of sums)."""
import ctypes as C

import numpy as np
import pytest

import host
from conftest import fields_err, rel_err
from pyugks_b200 import _lib, configs
from pyugks_b200.fused import FusedSolver

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-11


def oracle(case, steps):
    ora = host.OracleSim(case, "port")
    for _ in range(steps):
        ora.one_step()
    return ora


def check(gpu, ora):
    assert gpu.solve_state()[0]["status"] == 0
    assert fields_err(gpu.fields(), ora.fields()) < FP64_TOL
    for a, b in zip(gpu.interior_f(), ora.interior_f()):
        assert rel_err(a, b) < FP64_TOL


@pytest.mark.parametrize("scheme", ["vanLeer", "WENO5", "minmod"])
@pytest.mark.parametrize("n,nj,m", [(3, 4, 4), (5, 7, 8), (9, 6, 12), (4, 13, 16)])
def test_sizes(cuda, scheme, n, nj, m):
    """25, 81, 169 and 289 velocities (below one trip of a warp, and with
    remainders), block sides with every remainder of the strip width."""
    case = configs.cavity(n=n, nj=nj, m=m, vlim=4.0, flux_method=scheme, Kn=0.1, CFL=0.2)
    ora = oracle(case, 5)
    gpu = FusedSolver(case)
    gpu.step(5)
    check(gpu, ora)


@pytest.mark.parametrize("scheme", ["vanLeer", "WENO5"])
def test_warped(cuda, scheme):
    case = configs.warped_cavity(n=7, m=8, flux_method=scheme, CFL=0.2)
    ora = oracle(case, 5)
    gpu = FusedSolver(case)
    gpu.step(5)
    check(gpu, ora)


@pytest.mark.parametrize("m", [4, 8])
def test_grid_without_axes(cuda, m):
    """u_num = 0 in the block table: the Maxwellian of every velocity by exp
    instead of axis factors."""
    import torch
    case = configs.cavity(n=6, m=m, vlim=4.0, Kn=0.1, CFL=0.2)
    ora = oracle(case, 5)
    gpu = FusedSolver(case)
    structs = []
    for b in gpu.blocks:
        x = _lib.FusedBlock.from_buffer_copy(bytes(b.struct))
        x.d.u_num = x.d.v_num = 0
        structs.append(x)
    arr = (_lib.FusedBlock * len(structs))(*structs)
    assert gpu.lib.ugks_fused_layout(arr, len(structs), C.byref(gpu.sizes)) == 0
    assert gpu.sizes.max_axes == 0
    gpu.table = torch.from_numpy(np.frombuffer(bytes(arr), dtype=np.uint8).copy()).to(gpu.device)
    gpu.step(5)
    check(gpu, ora)
