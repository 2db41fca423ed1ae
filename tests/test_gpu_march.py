"""The streaming launcher operators (march.cu, stencil3.cu) at the edges of their thread mapping:
rows of whole vectors and odd rows, axes shorter than a segment, one column of vectors, sizes around
a block of 4 steps, and fields that are not 16-byte aligned.  Against the CPU FP64 oracle:
FP64 1e-12, FP32 1e-5 of the largest value (sums of at most 21 terms; FP32 inputs rounded first)."""
import numpy as np
import pytest
import torch

import oracle as O
import impact_b200 as I
from _util import rel_err

pytestmark = pytest.mark.gpu
SIZES = [(9, 9, 9), (10, 17, 12), (17, 9, 21), (13, 14, 75), (65, 33, 10), (38, 47, 18), (131, 19, 16)]


def _dev(a, f32, shift):
    """The array on the device, `shift` elements into its allocation."""
    t = torch.zeros(a.size + 8, dtype=torch.float32 if f32 else torch.float64, device="cuda")
    v = t[shift:shift + a.size]
    v.copy_(torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda())
    return v


@pytest.mark.parametrize("f32", [False, True], ids=["fp64", "fp32"])
@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "shifted"])
@pytest.mark.parametrize("N", SIZES, ids=lambda n: "x".join(str(v - 1) for v in n))
def test_streaming_operators_at_their_edges(N, shift, f32):
    og, ig = O.Grid(N, (1.0, 0.7, 1.3), (1, 0, 1)), I.Grid(N, (1.0, 0.7, 1.3), (1, 0, 1))
    tol, sfx, real = (1e-5, "_sp_", "f") if f32 else (1e-12, "_", "d")
    d = [("i", n + 7) for n in N]
    tab = lambda name, a: _dev(ig.tab[name][a], f32, 0)  # noqa: E731

    def call(name, ints, scalars, arrays, out):
        I.launchers.call(name + sfx, *ints, *[(real, v) for v in scalars], *[("p", t.data_ptr()) for t in arrays])
        torch.cuda.synchronize()
        return out.cpu().numpy().astype(np.float64).reshape(og.shape if out.numel() == og.zeros().size else -1)

    f, g, h = og.random(3), og.random(4), og.random(5)
    df, dg = _dev(f, f32, shift), _dev(g, f32, shift)
    for m in (1, 2, 3):
        out = _dev(og.zeros(), f32, shift)
        got = call("gradient_launcher", [("i", m), *d, ("i", 6), ("i", N[m - 1] + 1)], [], [df, tab("cG", m - 1), out], out)
        assert rel_err(og.interior(got), og.interior(og.gradient(m, f))) <= tol
        got = call("interpolate2_vel_pre_launcher", [("i", m), *d, ("i", 6), ("i", N[m - 1] + 1)], [],
                   [df, tab("cIup", m - 1), out], out)
        assert rel_err(og.interior(got), og.interior(og.interpolate_vel_pre(m, f))) <= tol
        for a in range(3):
            cid = 3 * (m - 1) + a + 1
            up, dn = ("cNuU", "cNuD") if a == m - 1 else ("cNpU", "cNpD")
            out = _dev(h, f32, shift)
            got = call("nonlinear_upwind_launcher", [("i", cid), *d, ("i", 7), ("i", N[a] + 1)], [],
                       [dg, df, out, tab(up, a), tab(dn, a)], out)
            assert rel_err(og.interior(got), og.interior(og.nonlinear_upwind(cid, g, f, h.copy()))) <= tol
        out = _dev(h, f32, shift)
        c = [tab("cuu" if a == m - 1 else "cpp", a) for a in range(3)]
        got = call("helmholtz_explicit_launcher", [("i", m), *d, ("i", 7), ("i", 7), ("i", 7)], [1e-3], [df, out, *c], out)
        assert rel_err(og.interior(got), og.interior(og.helmholtz(m, 1e-3, f, h.copy()))) <= tol
    vel = og.random(6, n=3)
    dv, out = _dev(vel, f32, shift), _dev(og.zeros(), f32, shift)
    got = call("divergence2_launcher", [*d, ("i", 6), ("i", 6), ("i", 6)], [], [dv, out, *[tab("cD", a) for a in range(3)]], out)
    assert rel_err(og.interior(got), og.interior(og.divergence2(vel[0], vel[1], vel[2]))) <= tol
    out = _dev(og.zeros(), f32, shift)
    got = call("jacobi_launcher", [("i", 1), *d, *[("i", n) for n in N], ("i", 3)], [0.8],
               [*[tab("cdg", a) for a in range(3)], df, dg, out], out)
    assert rel_err(og.interior(got), og.interior(og.jacobi(g.copy(), f.copy(), 1, 0.8, init_yes=False))) <= tol
    got = call("axpby_launcher", d, [0.5, -2.0], [df, dg, out], out)
    assert rel_err(og.interior(got), 0.5 * og.interior(f) - 2.0 * og.interior(g)) <= tol
