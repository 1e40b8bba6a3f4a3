# SPDX-License-Identifier: GPL-3.0-or-later
"""The acoustic substeps of an undecomposed domain take the points past its edges from the domain itself instead of from
filled halos. 3-D flows that vary along both directions, over terrain, with every pair of boundary kinds that the
substeps tell apart, alone and as members of one batch with a specified domain: bit-identical to the oracle, which fills
the halos before and between the substeps."""
import numpy as np
import pytest

import _oracle
from cases import lam_case
from cppwrf_b200 import Batch, capi
from test_parity_gpu import compare_all, run_pair

pytestmark = pytest.mark.gpu

P, S, O = capi.PERIODIC, capi.SYMMETRIC, capi.OPEN
KINDS = [(S, S), (P, P), (O, S), (S, O), (P, S), (S, P), (O, P), (P, O), (O, O)]


@pytest.mark.parametrize("bc", KINDS, ids=["%d-%d" % b for b in KINDS])
@pytest.mark.parametrize("nx,ny", [(13, 11), (34, 9)])
def test_boundary_kinds(bc, nx, ny):
    case = lam_case(nx=nx, ny=ny, nz=10, n_moist=2, n_scalars=2, seed=5, bc=bc)
    dom, orc = run_pair(case, 2)
    bad = compare_all(dom, orc, case)
    assert not bad, "\n".join(bad)


def test_batch_of_mixed_boundary_kinds():
    kinds = [(capi.SPECIFIED, capi.SPECIFIED), (P, S), (S, S), (O, P)]
    cases = [lam_case(nx=15 + 6 * m, ny=13 - m, nz=9 + 3 * m, n_moist=1, n_scalars=1, seed=20 + m, bc=bc)
             for m, bc in enumerate(kinds)]
    b = Batch([c.g for c in cases], [c.o for c in cases])
    for m, c in enumerate(cases):
        b.upload_case(m, c)
    b.step(2)
    for m, c in enumerate(cases):
        orc = _oracle.Oracle(c, pow_mode=_oracle.POW_OWN)
        orc.step(2)
        for name in capi.STATE_FIELDS + ["MUTS", "AL", "WW"]:
            assert np.array_equal(b.field(m, name).view(np.uint64), orc.array(name).view(np.uint64)), (m, name)
