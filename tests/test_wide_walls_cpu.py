"""The block table's launch of Cercignani-Lampis walls (ugks_fused_layout on the
host): present when a block of more than 1100 velocities has one."""
import ctypes as C

import pytest

from pyugks_b200 import _lib
from pyugks_b200 import defs as D
from test_layout_cpu import block, layout

CL = 2  # ugks_block_desc.reflect: Cercignani-Lampis


def walled(m, bc=D.ADSORBING, reflect=CL, **kw):
    x = block(m=m, **kw)
    x.bc_type[D.WEST] = bc
    x.d.reflect[D.WEST] = reflect
    return x


@pytest.mark.parametrize("x,present", [
    (walled(37), True), (walled(33), False), (walled(37, reflect=0), False), (walled(37, reflect=1), False),
    (walled(37, bc=D.DIFFUSE), False)])
def test_when_present(x, present):
    rc, z = layout([x])
    assert rc == 0
    assert (z.seg_method[z.n_segments - 1] == _lib.SEG_CL_WALLS) == present
    assert z.n_segments == (2 if present else 1)
    L = _lib.lib()
    assert L.ugks_step_launches(C.byref(z), 0) == (5 if present else 4)
    assert L.ugks_step_launches(C.byref(z), 1) == 7


def test_it_counts_among_the_segments():
    """20 velocity grids of one limiter, the widest with such a wall: 15 runs and it."""
    rc, z = layout([block(solve=k, m=9 + 2 * k) for k in range(19)] + [walled(49, solve=19)])
    assert rc == 0 and z.n_segments == 16
    assert z.seg_method[15] == _lib.SEG_CL_WALLS and z.seg_count[15] == z.n_wall
    assert sum(z.seg_count[k] for k in range(15)) == z.n_faces
    rc, z = layout([block(solve=k, m=9 + 2 * k) for k in range(20)])
    assert rc == 0 and z.n_segments == 16 and sum(z.seg_count) == z.n_faces
