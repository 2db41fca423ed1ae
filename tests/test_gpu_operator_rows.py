"""The FP32 operator's vector kernel has two forms: two rows per thread (tiles of 32 x 16 columns, the
tile's own points published from the z window, depth by the grid) in multigrid solves, one row (tiles
of 32 x 8) in solves with JOR sweeps.  Case.apply(op=2) runs the first on a case with a multigrid
hierarchy and the second on one without, created without coordinates.  Each against the oracle (1e-5 of
max|A x|: the rounding of input, weights and 33 products per point; an indexing error is of order
one), and against each other bit for bit: both sum a point's terms in the same order."""
import numpy as np
import pytest

import oracle as O
import impact_b200 as I

pytestmark = pytest.mark.gpu

# one row and one column over a tile, one short of it, an odd last pair of rows (its image row), tiles of
# 2 planes, ragged last steps, several tiles along each axis, the smallest grid
SIZES = [(32, 16, 8), (36, 17, 9), (28, 15, 34), (64, 31, 11), (8, 33, 131), (12, 47, 10), (8, 8, 8), (100, 41, 26),
         (64, 56, 102), (96, 48, 64)]


def _no_hierarchy(grid):
    """The grid's tables without its coordinates: a case that has no multigrid levels."""
    for a in range(3):
        grid.coeffs.xp[a] = None
        grid.coeffs.xu[a] = None
    return grid


@pytest.mark.parametrize("n", SIZES, ids=lambda n: "%dx%dx%d" % n)
def test_both_forms_of_the_fp32_operator(n):
    N, L = tuple(k + 1 for k in n), tuple(k / 32.0 for k in n)
    og = O.Grid(N, L, (0, 0, 0))
    x = og.random(23)
    want = og.interior(og.product_div_grad(x.copy()))
    got = []
    for grid, levels in ((I.Grid(N, L, (0, 0, 0)), True), (_no_hierarchy(I.Grid(N, L, (0, 0, 0))), False)):
        case = I.Case(grid, precision=1)
        assert (case.mg_levels > 0) == levels
        case.upload("pre", x)
        case.apply("pre", "res", op=2)
        got.append(og.interior(case.download("res")).copy())
        assert np.abs(got[-1] - want).max() <= 1e-5 * np.abs(want).max()
        case.close()
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("n", [(32, 24, 40), (40, 24, 24), (48, 40, 16)], ids=lambda n: "%dx%dx%d" % n)
def test_two_row_sums_carry_a_multigrid_solve(n):
    """alpha and omega come from the two-row kernel's partial sums: a row or plane left out of them would spoil
    every step of BiCGstab.  The mixed solve's FP32 iterations must then reach the tolerance in about as many
    as the FP64 solve's (one more per refinement for the FP32 rounding)."""
    N, L = tuple(k + 1 for k in n), tuple(k / 32.0 for k in n)
    og = O.Grid(N, L, (0, 0, 0))
    b = og.product_div_grad(og.random(24).copy())
    its = []
    for precision in (0, 1):
        case = I.Case(I.Grid(N, L, (0, 0, 0)), precision=precision)
        case.upload("res", b)
        r = case.poisson("res", "pre", I.solver_params(precond=1, mg_down=3, mg_up=3, mg_bottom=3, tol_rel=1e-8, init_yes=1,
                                                       max_it=60 if precision == 0 else 20, inner_tol_rel=1e-3, inner_max_it=60))
        assert r.status == 0
        its.append((r.iterations, r.inner_iterations))
        case.close()
    assert its[1][1] <= its[0][0] + 2 * its[1][0]
