"""Lists of many cases: the operator's tiles hold several units of summation there (one when a case is
alone), so a case's sums, and with them every bit of its step, must not depend on the batch."""
import numpy as np
import pytest

import impact_b200 as I
from impact_b200 import geometry as G

pytestmark = pytest.mark.gpu

# whole units and ragged last ones along z, rows of 4 and of 2, an odd second axis
SIZES = [(32, 32, 64), (36, 28, 52), (40, 33, 47), (30, 24, 38)]
FIELDS = ("vel1", "vel2", "vel3", "pre")


def _case(n, precision):
    g = I.Grid(tuple(k + 1 for k in n), tuple(k / 32.0 for k in n))
    c = I.Case(g, precision=precision)
    c.set_labels(G.straight_vessel(g))
    return c


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_tiles_of_several_units_give_the_sums_of_a_case_alone(precision):
    p = I.step_params(Re=200.0, U0=1.0, tol_rel=1e-8, omega=0.8, precond=1, mg_down=3, mg_up=3, mg_bottom=3, tile_kc=64,
                      max_it=200 if precision == 0 else 40, inner_tol_rel=3e-3)
    made = [_case(n, precision) for n in SIZES * 15]
    batch = I.Batch(made)
    batch.step([p] * len(made))
    for q, n in enumerate(SIZES):
        one = _case(n, precision)
        one.step(p, 1)
        for f in FIELDS:
            want = one.download(f)
            assert np.isfinite(want).all()
            assert np.array_equal(made[q].download(f), want), (n, f)
            assert np.array_equal(made[len(made) - len(SIZES) + q].download(f), want), (n, f)
        one.close()
    batch.close()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("sweeps", [2, 3, 4])
def test_fused_jor_sweeps_in_a_batch_of_uneven_cases(sweeps, precision):
    """The JOR preconditioner's fused sweeps (one z-marching kernel over the whole list) on uneven cases, odd rows
    among them: every case must end bit for bit as alone."""
    p = I.step_params(Re=200.0, U0=1.0, tol_rel=1e-8, omega=0.8, precond=0, n_sweeps=sweeps, check_every=4,
                      max_it=2000 if precision == 0 else 40, inner_max_it=4000, inner_tol_rel=3e-3)
    sizes = [(24, 20, 32), (19, 23, 28), (33, 16, 21), (16, 16, 16)]
    made = [_case(n, precision) for n in sizes]
    batch = I.Batch(made)
    batch.step([p] * len(made))
    for c, n in zip(made, sizes):
        one = _case(n, precision)
        one.step(p, 1)
        assert all(s == 0 for s in one.state.poisson_status)
        for f in FIELDS:
            assert np.array_equal(c.download(f), one.download(f)), (n, f)
        one.close()
    batch.close()
