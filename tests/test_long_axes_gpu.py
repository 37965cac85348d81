"""Velocity grids with more than 512 axis nodes (a few nodes in u, hundreds in v, and
the reverse), on either side of that count, alone and beside a small grid: the FP64
kernels then take exponentials instead of axis factors, the mixed ones keep longer
tables.  Against the oracle, with the tolerances of the fused path's other parity
tests (FP64 1e-11, mixed 1e-5)."""
import pytest

import host
from conftest import fields_err, rel_err
from pyugks_b200 import configs
from pyugks_b200.fused import FusedSolver

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-11, "mixed": 1e-5}


def case(u, v, scheme):
    c = configs.cavity(n=3, nj=4, m=8, vlim=4.0, flux_method=scheme, Kn=0.3, CFL=0.2)
    c["quad"] = dict(c["quad"], u_num=u, v_num=v)
    return c


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("scheme", ["vanLeer", "WENO5", "minmod"])
@pytest.mark.parametrize("u,v", [(8, 500), (8, 504), (504, 8), (4, 800)])
def test_long_axes(cuda, u, v, scheme, precision):
    """510, 514 (both ways) and 806 nodes: u // 4 * 4 + 1 and v // 4 * 4 + 1."""
    cases = [case(u, v, scheme), case(8, 8, scheme)]
    gpu = FusedSolver(cases, precision=precision)
    gpu.step(3)
    for k, c in enumerate(cases):
        ora = host.OracleSim(c, "port")
        for _ in range(3):
            ora.one_step()
        assert gpu.solve_state()[k]["status"] == 0
        assert fields_err(gpu.fields(k), ora.fields()) < TOL[precision]
        assert rel_err(gpu.interior_f(k)[0], ora.interior_f()[0]) < TOL[precision]
