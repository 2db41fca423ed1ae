"""Launch shapes of the streaming passes (csrc/shape.h, compiled here for the host) and the registers
of their kernels: a small grid may not be left to a few long threads or blocks, a large one not to a
nearly empty last wave, and no kernel of the one-axis passes may spill."""
import ctypes as C
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpu-impact-ct_b200", "csrc")
SMS = 148


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    out = tmp_path_factory.mktemp("shape") / "libshape_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, os.path.join(ROOT, "tests", "shape_host.cpp"),
                    "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    lib.host_march_seg.restype, lib.host_march_seg.argtypes = C.c_int, [C.c_longlong] + [C.c_int] * 4
    lib.host_tri_depth.restype, lib.host_tri_depth.argtypes = C.c_int, [C.c_double, C.c_int, C.c_double, C.c_int]
    lib.host_stack.restype, lib.host_stack.argtypes = None, [C.POINTER(C.c_int)] + [C.c_int] * 5 + [C.POINTER(C.c_int)] * 2
    return lib


@pytest.mark.parametrize("per_sm,most", [(320, 8), (256, 16)], ids=["y-z", "x"])
@pytest.mark.parametrize("vector", [1, 2, 4])
@pytest.mark.parametrize("n", [8, 9, 16, 24, 33, 48, 56, 57, 64, 81, 128, 256])
def test_a_marching_pass_fills_the_device_before_it_lengthens_its_segments(shape, n, vector, per_sm, most):
    threads, na = -(-n // vector) * n, n
    seg = shape.host_march_seg(threads, na, SMS, per_sm, most)
    assert 1 <= seg <= min(most, na)
    launched = threads * -(-na // seg)
    assert seg == 1 or launched >= SMS * per_sm
    assert seg == most or 2 * seg > na or threads * na < SMS * per_sm * 2 * seg


def test_a_three_axis_pass_prefers_one_full_wave(shape):
    # tiles of 32 x 16 points of two doubles: one wave of two blocks per SM
    for n, kz in ((112, 12), (128, 16), (160, 32), (192, 48)):
        gxy = -(-n // 32) * -(-n // 16)
        assert shape.host_tri_depth(gxy, n, SMS, 1) == kz
        assert SMS < gxy * -(-n // kz) <= 2 * SMS


@pytest.mark.parametrize("vec", [0, 1])
@pytest.mark.parametrize("n", [8, 16, 24, 48, 64])
def test_a_three_axis_pass_on_a_small_grid_takes_shallow_blocks(shape, n, vec):
    gxy = -(-n // 32) * -(-n // (16 if vec else 8))
    kz = shape.host_tri_depth(gxy, n, SMS, vec)
    assert gxy * -(-n // kz) >= min(SMS / 2, gxy * n)


def test_long_axes_stay_within_the_launch_limit(shape):
    for n in (65535, 65536, 600_000, 3_000_000, 20_000_000):
        for threads in (16, 32, 64):
            assert -(-n // shape.host_march_seg(threads, n, SMS, 320, 8)) <= 65535
        for vec in (0, 1):
            assert -(-n // shape.host_tri_depth(1, n, SMS, vec)) <= 65535


@pytest.mark.parametrize("share", [1.0, 0.25, 0.001])
def test_depths_of_a_batch_grow_as_its_share_shrinks(shape, share):
    assert shape.host_tri_depth(8, 64, SMS * share, 1) >= shape.host_tri_depth(8, 64, SMS, 1)


def _stacked(shape, sizes, rows, kc, slots, step):
    arr = C.c_int * len(sizes)
    ks, depth = arr(), arr()
    shape.host_stack(arr(*sizes), len(sizes), rows, kc, slots, step, ks, depth)
    return list(ks), list(depth)


def _planes(sizes, depths, rows):
    """Planes marched by a list's tiles, with the 8 planes' time of each tile's prologue."""
    return sum(-(-n // 32) * -(-n // rows) * sum(min(d, 2 * n - k) + 8 for k in range(0, 2 * n, d)) for n, d in zip(sizes, depths))


UNEVEN = [32, 40, 40, 48, 56, 64, 64, 72, 80, 88, 96, 96, 104, 112, 120, 136, 144, 152]
KERNELS = [(8, 296, 4), (16, 296, 2), (16, 592, 2)]  # FP64 operator, FP64 outer residual, FP32 operator


@pytest.mark.parametrize("rows,slots,step", KERNELS, ids=["fp64", "residual", "fp32"])
def test_a_batch_does_not_pay_for_the_shallow_tiles_of_its_cases_alone(shape, rows, slots, step):
    sizes = 3 * UNEVEN
    ks, depth = _stacked(shape, sizes, rows, 64, slots, step)
    deep, alone = _planes(sizes, [64] * len(sizes), rows), _planes(sizes, ks, rows)
    assert alone > 1.1 * deep
    assert _planes(sizes, depth, rows) - deep <= 0.25 * (alone - deep)  # (the rest: units that do not divide 64, the last wave)
    for n, u, d in zip(sizes, ks, depth):
        assert d % u == 0 and d <= 64
        assert u == _stacked(shape, [n], rows, 64, slots, step)[0][0]  # the unit is the grid's own


@pytest.mark.parametrize("rows,slots,step", KERNELS, ids=["fp64", "residual", "fp32"])
@pytest.mark.parametrize("kc", [1, 5, 8, 12, 30, 64])
@pytest.mark.parametrize("n", [8, 33, 64, 160])
def test_a_case_alone_keeps_one_unit_per_tile(shape, n, kc, rows, slots, step):
    ks, depth = _stacked(shape, [n], rows, kc, slots, step)
    assert depth == ks and 1 <= ks[0] <= kc


@pytest.mark.parametrize("kc", [1, 5, 8, 12, 30, 64])
def test_tiles_of_several_units_hold_whole_steps(shape, kc):
    for rows, slots, step in KERNELS:
        ks, depth = _stacked(shape, UNEVEN, rows, kc, slots, step)
        for u, d in zip(ks, depth):
            assert d == u or (u % step == 0 and d % u == 0 and d <= kc)


def test_a_coarse_tail_takes_no_cluster_that_the_device_cannot_hold(shape):
    def f(ntails, held, fitted=8):
        return shape.host_tail_cluster(ntails, (C.c_int * 3)(*held), fitted)
    whole = (74, 33, 15)
    assert [f(n, whole) for n in (1, 15, 16, 33, 34, 74, 75)] == [8, 8, 4, 4, 2, 2, 1]
    assert [f(1, whole, fitted) for fitted in (8, 4, 2, 1)] == [8, 4, 2, 1]
    assert [f(1, part) for part in ((4, 2, 0), (4, 0, 0), (0, 0, 0))] == [4, 2, 1]


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_one_axis_kernels_do_not_spill(tmp_path):
    r = subprocess.run(["nvcc", "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                        "-gencode", "arch=compute_100a,code=sm_100a", "-Xptxas", "-v", "-cubin", "-o", str(tmp_path / "march.cubin"),
                        os.path.join(CSRC, "march.cu")], capture_output=True, text=True, check=True)
    kernels = re.findall(r"Compiling entry function '(\S*k_march_\S*)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads", r.stderr, re.S)
    assert len(kernels) == 32  # 4 operators, 2 orientations, vectors and points, 2 types
    assert [k for k in kernels if k[1:] != ("0", "0")] == []
