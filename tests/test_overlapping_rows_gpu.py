# SPDX-License-Identifier: GPL-3.0-or-later
"""Specified domains of fewer than 8 points along a direction, down to the smallest that is accepted: the relaxation rows
of opposite sides overlap, and a point takes the terms of every row it lies in. Bit-identical to the oracle, which adds
them side by side."""
import pytest

from cases import lam_case
from cppwrf_b200 import Batch, capi
from test_parity_gpu import compare_all, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(4, 4), (4, 9), (9, 4), (5, 6), (6, 5), (7, 7), (7, 8), (8, 7), (8, 8), (6, 23), (23, 7)])
def test_small_specified_domain(nx, ny):
    case = lam_case(nx=nx, ny=ny, nz=8, n_moist=2, n_scalars=2, seed=nx + 10 * ny)
    dom, orc = run_pair(case, 2)
    bad = compare_all(dom, orc, case)
    assert not bad, "\n".join(bad)


def test_small_members_of_a_batch():
    import _oracle
    import numpy as np

    cases = [lam_case(nx=nx, ny=ny, nz=9, n_moist=1, n_scalars=1, seed=nx) for nx, ny in ((6, 9), (20, 14), (12, 5))]
    b = Batch([c.g for c in cases], [c.o for c in cases])
    for m, c in enumerate(cases):
        b.upload_case(m, c)
    b.step(2)
    for m, c in enumerate(cases):
        orc = _oracle.Oracle(c, pow_mode=_oracle.POW_OWN)
        orc.step(2)
        for name in capi.STATE_FIELDS:
            assert np.array_equal(b.field(m, name).view(np.uint64), orc.array(name).view(np.uint64)), (m, name)


@pytest.mark.parametrize("nx,ny,px,py", [(14, 6, 2, 1), (7, 13, 1, 2)])
def test_small_side_of_a_decomposed_domain(nx, ny, px, py):
    from test_decomp_gpu import compare, run_both

    case = lam_case(nx=nx, ny=ny, nz=8, n_moist=2, n_scalars=2, seed=nx)
    dec, dom = run_both(case, px, py, 2)
    bad = compare(dec, dom, case)
    assert not bad, "\n".join(bad)
