"""The FP64 face pass with every stage of its asynchronous copies refilled several
times (1089 velocities: 35 trips of a warp over 2, 3 and 5 stages): the oracle's
values (tolerance of the fused path's other parity tests) and, over again, the same
bits."""
import numpy as np
import pytest

import host
from conftest import fields_err, rel_err
from pyugks_b200 import configs
from pyugks_b200.fused import FusedSolver

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-11


@pytest.mark.parametrize("scheme", ["vanLeer", "WENO5", "minmod"])
def test_refilled_stages(cuda, scheme):
    case = configs.cavity(n=9, nj=14, m=32, vlim=5.0, flux_method=scheme, Kn=0.1, CFL=0.3)
    ora = host.OracleSim(case, "port")
    for _ in range(4):
        ora.one_step()
    runs = []
    for _ in range(8):
        gpu = FusedSolver(case)
        gpu.step(4)
        b = gpu.blocks[0]
        runs.append([t.cpu().numpy() for t in (b.f, b.flux_S, b.flux_W, b.flux_macro_S, b.flux_macro_W)])
        assert fields_err(gpu.fields(), ora.fields()) < FP64_TOL
        assert rel_err(gpu.interior_f()[0], ora.interior_f()[0]) < FP64_TOL
    for r in runs[1:]:
        for x, y in zip(r, runs[0]):
            np.testing.assert_array_equal(x, y)
