"""The one-block coarse tail of the V-cycle (k_lv_tail) at the edges of its thread mapping and of
its shared memory: levels with more columns than threads, one plane or a partial segment per
thread, two-point axes, and tables too long to be staged.  Like every fused phase it must give the
iterate of the one-launch-per-phase schedule (which has no tail) bit for bit; so must the JOR
preconditioner's fused sweeps."""
import numpy as np
import pytest

import impact_b200 as I
from impact_b200 import geometry as G

pytestmark = pytest.mark.gpu

GRIDS = [((33, 33, 9), (1.0, 1.0, 0.25), (0, 0, 0)),      # first tail level 32 x 32 x 8: 1024 columns
         ((49, 25, 13), (1.0, 0.5, 0.25), (1, 0, 1)),     # 48 x 24 x 12, z rows differ
         ((9, 9, 1201), (0.1, 0.1, 15.0), (0, 0, 0)),     # 4 x 4 x 600 and coarser: tables of 6000 values
         ((21, 13, 37), (1.0, 0.6, 1.8), (0, 0, 0)),      # 20 x 12 x 36 -> 5 x 3 x 9
         ((9, 9, 9), (1.0, 1.0, 1.0), (0, 0, 0))]         # 8 x 8 x 8 -> 2 x 2 x 2


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("gi", range(len(GRIDS)), ids=["32x32x8", "48x24x12-xz", "8x8x1200", "20x12x36", "8x8x8"])
@pytest.mark.parametrize("sw", [(1, 1, 1), (2, 3, 1), (3, 2, 3)], ids=lambda s: "%d%d%d" % s)
def test_coarse_tail_equals_one_launch_per_phase(gi, sw, precision):
    g = I.Grid(*GRIDS[gi])
    case = I.Case(g, precision=precision)
    case.upload("res", np.random.default_rng(31).uniform(-1.0, 1.0, g.shape))
    out = []
    for unfused in (1, 0):
        case.precond("res", "pre", I.solver_params(precond=1, mg_down=sw[0], mg_up=sw[1], mg_bottom=sw[2],
                                                   smooth_unfused=unfused))
        out.append(g.interior(case.download("pre")).copy())
    assert np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1])
    case.close()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("N", [(9, 9, 9), (33, 29, 41), (60, 48, 84), (65, 65, 33)], ids=lambda n: "x".join(str(v - 1) for v in n))
@pytest.mark.parametrize("sweeps", [1, 2, 3, 4, 5])
def test_fused_jor_preconditioner_equals_one_sweep_per_launch(sweeps, N, precision):
    g = I.Grid(N, (1.0, 0.8, 1.3), (0, 0, int(N[0] == 33)))
    case = I.Case(g, precision=precision)
    case.upload("res", np.random.default_rng(32).uniform(-1.0, 1.0, g.shape))
    out = []
    for unfused in (1, 0):
        case.precond("res", "pre", I.solver_params(precond=0, n_sweeps=sweeps, smooth_unfused=unfused))
        out.append(g.interior(case.download("pre")).copy())
    assert np.array_equal(out[0], out[1])
    case.close()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [(26, 26, 22), (38, 38, 10), (26, 26, 34), (10, 38, 38)], ids=lambda n: "%dx%dx%d" % n)
def test_chebyshev_tail_cut_into_slabs_equals_one_block(n, precision):
    """Alone, a case's Chebyshev tail is cut into z slabs over a cluster of blocks (here with a short
    last slab, fewer planes than blocks, two levels in FP32); in a batch of more tails than half the
    device's 148 SMs every tail runs in one block.  Both must give the same step bit for bit."""
    def case():
        g = I.Grid(tuple(k + 1 for k in n), tuple(k / 26.0 for k in n))
        c = I.Case(g, precision=precision)
        c.set_labels(G.straight_vessel(g))
        return c
    p = I.step_params(Re=200.0, U0=1.0, tol_rel=1e-8, omega=0.8, precond=1, mg_down=3, mg_up=3, mg_bottom=3,
                      max_it=200 if precision == 0 else 40, inner_tol_rel=3e-3, bottom_cheb=12)
    fields = ("vel1", "vel2", "vel3", "pre")
    one = case()
    one.step(p, 2)
    made = [case() for _ in range(80)]
    batch = I.Batch(made)
    for _ in range(2):
        batch.step([p] * len(made))
    for f in fields:
        want = one.download(f)
        assert np.isfinite(want).all()
        assert np.array_equal(made[0].download(f), want) and np.array_equal(made[-1].download(f), want), f
    batch.close()
    one.close()
