"""The ways a step is launched (programmatic launches for small tables, plain ones
with the mixed walls on a side stream for large), the mixed passes at the edges of
their work, and the residual over more cells than its CTA has threads."""
import numpy as np
import pytest

import host
from conftest import rel_err
from pyugks_b200 import configs
from pyugks_b200.fused import FusedSolver

pytestmark = pytest.mark.gpu

# deviations in FP32: every velocity takes some 16 roundings a step (stencil,
# slopes, flux, update), each of at most 2^-24 of the deviation, itself below f
MIXED_TOL = 16 * 5 * 2.0 ** -24


def small():
    return [configs.cavity(n=7, nj=5, m=8, vlim=4.0, flux_method="WENO5", Kn=0.1),
            configs.cavity(n=6, nj=9, m=12, vlim=4.0, flux_method="minmod", Kn=0.3, CFL=0.4),
            configs.channel(nblocks=2, n=6, m=8)]


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_same_bits_from_either_launch(cuda, precision, captured):
    """Solves of three limiters (several launches of a face pass) in a small table
    and beside a solve that takes the table over the line: the same bits."""
    def run(cases):
        s = FusedSolver(cases, precision=precision)
        if captured:
            s.capture(3)
            s.replay()
            s.replay()
        else:
            s.step(6)
        return s
    few, many = run(small()), run(small() + [configs.cavity(n=70, m=32, vlim=4.0)])
    for k in range(3):
        assert few.solve_state()[k]["status"] == 0 and few.solve_state()[k]["steps"] == 6
        assert few.solve_state()[k]["dt"] == many.solve_state()[k]["dt"]
        for a, b in zip(few.interior_f(k), many.interior_f(k)):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("scheme", ["vanLeer", "WENO5", "minmod"])
@pytest.mark.parametrize("n,nj,m", [(3, 4, 4), (5, 7, 8), (9, 6, 12), (4, 13, 16)])
def test_mixed_sizes(cuda, scheme, n, nj, m):
    """13, 41, 85 and 145 velocity pairs, block sides with every remainder."""
    case = configs.cavity(n=n, nj=nj, m=m, vlim=4.0, flux_method=scheme, Kn=0.1, CFL=0.2)
    ora = host.OracleSim(case, "port")
    for _ in range(5):
        ora.one_step()
    gpu = FusedSolver(case, precision="mixed")
    gpu.step(5)
    assert gpu.solve_state()[0]["status"] == 0
    for a, b in zip(gpu.interior_f(), ora.interior_f()):
        assert rel_err(a, b) < MIXED_TOL


@pytest.mark.parametrize("n,nj", [(3, 5), (31, 33), (32, 32), (36, 35)])
def test_residual_sizes(cuda, n, nj):
    """15, 1023, 1024 and 1260 cells against the definition."""
    gpu = FusedSolver(configs.cavity(n=n, nj=nj, m=8, vlim=4.0, Kn=0.1))
    gpu.step(3)
    gpu.compute_residual()
    got = gpu.solve_state()[0]["residual"]
    p, o = (t.cpu().numpy().reshape(n * nj, 4) for t in (gpu.blocks[0].macro, gpu.blocks[0].prim_old))
    want = np.sqrt(n * nj * np.sum((p - o) ** 2, axis=0)) / np.sum(np.abs(p), axis=0)
    # sums of n nj positive terms: their order is worth (n nj) 2^-53 at most
    np.testing.assert_allclose(got, want, rtol=4 * n * nj * 2.0 ** -53)
