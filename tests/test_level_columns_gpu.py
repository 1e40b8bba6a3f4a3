# SPDX-License-Identifier: GPL-3.0-or-later
"""The column kernels that run one thread per column and level, at the sizes where their blocks change: level counts
around whole warps, the smallest and the largest level counts (from nz = 124 on a block holds fewer columns), column
counts around a block's width, and domains on both sides of the size from which the preparation and finish kernels run
in blocks of whole rows. The FP64 form equals the oracle bit for bit; every autotuned shape gives the same bits."""
import numpy as np
import pytest

from cppwrf_b200 import Batch, Domain, capi
from cases import golden_config, ideal_case, lam_case
from test_parity_gpu import compare_all, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(7, 8, 3), (8, 7, 7), (9, 10, 3), (10, 9, 7), (15, 9, 30), (16, 8, 31), (16, 9, 31),
                                      (17, 8, 32), (17, 9, 32), (9, 8, 63), (9, 9, 63), (23, 7, 64), (23, 9, 64), (12, 8, 123),
                                      (12, 9, 123), (11, 9, 126)])
def test_lam_levels_and_widths(nx, ny, nz):
    case = lam_case(nx=nx, ny=ny, nz=nz, n_moist=2, n_scalars=2, seed=nx + nz)
    dom, orc = run_pair(case, 2)
    bad = compare_all(dom, orc, case, names=capi.STATE_FIELDS)
    assert not bad, "\n".join(bad)


@pytest.mark.parametrize("nx,nz", [(33, 100), (40, 124), (31, 126)])
def test_ideal_tall_domains(nx, nz):
    case = ideal_case(dict(golden_config("warm_bubble"), nx=nx, nz=nz, ztop=100.0 * nz))
    dom, orc = run_pair(case, 2)
    bad = compare_all(dom, orc, case, names=capi.STATE_FIELDS)
    assert not bad, "\n".join(bad)


@pytest.mark.parametrize("ny", [246, 252])
def test_both_sides_of_the_whole_row_blocks(ny):
    """31 columns (with their last face) are one block of whole rows per row: 247 and 253 of them."""
    case = lam_case(nx=30, ny=ny, nz=8, n_moist=1, n_scalars=1, seed=2)
    dom, orc = run_pair(case, 1)
    bad = compare_all(dom, orc, case, names=capi.STATE_FIELDS)
    assert not bad, "\n".join(bad)


@pytest.mark.parametrize("ny", [108, 115, 150])
def test_around_the_waves_of_the_level_thread_form(ny):
    """At 61 w levels an SM holds one level-thread block: 4 (ny + 1) blocks are 3, 4 and 5 waves, where k_ss_prep, then
    k_ls_prep too, run in rows."""
    case = lam_case(nx=30, ny=ny, nz=60, n_moist=1, n_scalars=1, seed=6)
    dom, orc = run_pair(case, 1)
    bad = compare_all(dom, orc, case, names=capi.STATE_FIELDS)
    assert not bad, "\n".join(bad)


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("nz", [20, 70, 126])
def test_every_tuned_shape_gives_the_same_bits(nz, precision):
    case = lam_case(nx=21, ny=11, nz=nz, n_moist=1, n_scalars=1, seed=nz, precision=precision)
    a = Domain(case.g, case.o).upload_case(case).set_autotune(True).step(6)
    b = Domain(case.g, case.o).upload_case(case).step(6)
    for name in capi.STATE_FIELDS + ["Q_2"]:
        assert np.array_equal(a.field(name).view(np.uint64), b.field(name).view(np.uint64)), name


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED], ids=["fp64", "mixed"])
def test_every_tuned_shape_gives_the_same_bits_in_a_batch(precision):
    """Members of uneven level counts in blocks sized for the tallest one; the batch untuned, tuned, and its members alone."""
    cases = [lam_case(nx=nx, ny=9, nz=nz, n_moist=2, n_scalars=2, seed=nz, precision=precision)
             for nx, nz in ((21, 12), (14, 70), (33, 31))]
    a, b = (Batch([c.g for c in cases], [c.o for c in cases]) for _ in range(2))
    for m, c in enumerate(cases):
        a.upload_case(m, c)
        b.upload_case(m, c)
    a.set_autotune(True).step(6)
    b.step(6)
    for m, c in enumerate(cases):
        d = Domain(c.g, c.o).upload_case(c).step(6)
        for name in capi.STATE_FIELDS + ["Q_2"]:
            x = d.field(name).view(np.uint64)
            assert np.array_equal(a.field(m, name).view(np.uint64), x), (m, name)
            assert np.array_equal(b.field(m, name).view(np.uint64), x), (m, name)


@pytest.mark.parametrize("nz", [61, 70, 124, 126])
def test_reported_shape_is_the_one_that_ran(nz):
    """Where a shape's block does not fit, the kernel runs (and the tuner reports) another one: k_ac's 16 columns above 61
    levels and its 8 above 123, the level-thread form of the other column kernels above 123. The tuner measures no shape
    that did not run, however often it is asked."""
    case = lam_case(nx=12, ny=9, nz=nz, n_moist=1, n_scalars=1, seed=4)
    d = Domain(case.g, case.o).upload_case(case)
    for _ in range(4):
        d.set_autotune(True).step(6)
        assert d.autotune_choice("k_ac") in ((0, 1, 2) if nz <= 61 else (0, 2) if nz <= 123 else (2,))
        for k in ("k_ls_prep", "k_ss_prep", "k_finish"):
            assert d.autotune_choice(k) in ((0, 1, 2) if nz <= 123 else (0, 1)), k
