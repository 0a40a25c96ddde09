"""GPU: the FP64 far field on the int8 tensor cores in whole FMMs: strengths at the ends of the double
range, and the switch between them and cuBLAS."""
import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_fmm import fmm_case, run_fmm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return torch


# LapPGrad with double layer, Stokes, PVel (scaled densities)
@pytest.mark.parametrize("shift", [-1000, 960])
@pytest.mark.parametrize("kernel,max_pts", [(1, 60), (8, 60), (128, 150)])
def test_strengths_at_the_ends_of_the_double_range(torch_cuda, kernel, max_pts, shift):
    """Strengths times a power of two give results times that power: the same bits but for values
    below 2^-1022.  Those are at least 2^-22 below the strengths and are rounded at 2^-1074, 2^-74 of
    the strengths; the pseudo-inverses' factors of up to 1e8 (2^27) leave 2^-47 = 7e-15."""
    pts, slv, dlv, td = fmm_case(kernel, 6000, seed=90 + kernel)
    f, ref = run_fmm(kernel, 8, max_pts, pts, slv, dlv, td)
    g, got = run_fmm(kernel, 8, max_pts, pts, np.ldexp(slv, shift), None if dlv is None else np.ldexp(dlv, shift), td)
    assert np.isfinite(got).all()
    assert rel_l2(np.ldexp(got, -shift), ref) < 1e-14


@pytest.mark.parametrize("kernel,max_pts", [(1, 60), (8, 60)])
def test_every_handle_reads_the_switch(torch_cuda, monkeypatch, kernel, max_pts):
    """STKFMM_F64_I8 decides for the handle that is set up, not for all that share its operators: with
    all earlier handles alive, "1" and "0" give their own bits (both paths repeat theirs) each time."""
    pts, slv, dlv, td = fmm_case(kernel, 6000, seed=100 + kernel)
    handles, res = [], []
    for mode in ("0", "1", "0", "1"):
        monkeypatch.setenv("STKFMM_F64_I8", mode)
        f, out = run_fmm(kernel, 8, max_pts, pts, slv, dlv, td)
        handles.append(f)
        res.append(out)
    assert (res[0] != res[1]).any()
    np.testing.assert_array_equal(res[0], res[2])
    np.testing.assert_array_equal(res[1], res[3])
    # the first handle again, its tree set up anew under the other mode, and back
    for mode, want in (("1", 1), ("0", 0)):
        monkeypatch.setenv("STKFMM_F64_I8", mode)
        handles[0].setup_tree(kernel)
        out = np.zeros_like(res[0])
        handles[0].evaluate_fmm(kernel, slv, out, dlv)
        np.testing.assert_array_equal(out, res[want])


def used_bytes(torch):
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


# Stokes' translations in mixed precision: no int8 products at all; LapPGrad: the M2L's factors stay out
@pytest.mark.parametrize("kernel,extra", [(8, 0), (1, 64 << 20)])
def test_mixed_handles_hold_no_digits_they_do_not_use(torch_cuda, monkeypatch, kernel, extra):
    """Device memory of a handle's first mixed evaluation, with the int8 products on and off.  The
    operators' digits are 7 bytes a value: m2m, l2l (N x 8N) and four of at most N x N, 20 N^2 values,
    N = 296 for LapPGrad at p = 8 (12 MB), rounded up to blocks; the rest is the operand of a product."""
    import gc
    pts, slv, dlv, td = fmm_case(kernel, 6000, seed=110)
    run_fmm(kernel, 8, 60, pts, slv, dlv, td, prec=1)  # libraries and kernels are loaded
    used = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("STKFMM_F64_I8", mode)
        gc.collect()
        before = used_bytes(torch_cuda)
        f, _ = run_fmm(kernel, 8, 60, pts, slv, dlv, td, prec=1)
        used[mode] = used_bytes(torch_cuda) - before
        del f
    assert used["1"] <= used["0"] + extra + (8 << 20), used


@pytest.mark.parametrize("kernel,max_pts", [(1, 60), (8, 60), (128, 150)])
def test_precision_switched_between_evaluations(torch_cuda, kernel, max_pts):
    """One handle, mixed - FP64 - mixed - FP64: the bits of handles that were made in that precision."""
    pts, slv, dlv, td = fmm_case(kernel, 6000, seed=120 + kernel)
    f, _ = run_fmm(kernel, 8, max_pts, pts, slv, dlv, td, prec=1)
    fresh = [run_fmm(kernel, 8, max_pts, pts, slv, dlv, td, prec=prec) for prec in (0, 1)]
    for prec in (1, 0, 1, 0):
        f.set_precision(prec)
        out = np.zeros((len(pts), td))
        f.evaluate_fmm(kernel, slv, out, dlv)
        np.testing.assert_array_equal(out, fresh[prec][1])


# all digits but few, the operators' but not the factors', and somewhat more
@pytest.mark.parametrize("slack_mb", [40, 130, 250])
def test_set_up_where_the_digits_leave_no_room(torch_cuda, monkeypatch, slack_mb):
    """With the device memory that a handle needs without digits, and some of what they would take, a
    handle is set up and gives the sums: what runs without the int8 products runs with them on.  Their
    difference from cuBLAS is below the noise of such an FMM, 1e-9 (its error at p = 8 is 1e-6)."""
    import gc
    torch = torch_cuda
    pts, slv, _, td = fmm_case(8, 6000, seed=130)
    monkeypatch.setenv("STKFMM_F64_I8", "0")
    keep, ref = run_fmm(8, 8, 60, pts, slv, None, td)  # the operators stay
    gc.collect()
    torch.cuda.empty_cache()
    before = used_bytes(torch)
    f, _ = run_fmm(8, 8, 60, pts, slv, None, td)
    need = used_bytes(torch) - before
    del f
    gc.collect()
    monkeypatch.setenv("STKFMM_F64_I8", "1")
    hog = torch.empty(torch.cuda.mem_get_info()[0] - need - (slack_mb << 20), dtype=torch.uint8, device="cuda")
    try:
        f, out = run_fmm(8, 8, 60, pts, slv, None, td)
        assert rel_l2(out, ref) < 1e-9
        del f
    finally:
        del hog
        torch.cuda.empty_cache()
    # with room again the digits are made
    f, out = run_fmm(8, 8, 60, pts, slv, None, td)
    assert (out != ref).any() and rel_l2(out, ref) < 1e-9


def test_a_given_up_wait_is_an_error(torch_cuda):
    """The code that a tensor-core kernel leaves when a pipeline wait gives up, put there by a hook: the
    next call that looks (a host evaluation, last_kernel_ms) fails once, of the wall for every sub-FMM;
    set_up of a new tree clears it."""
    import stkfmm_b200 as S
    from stkfmm_b200 import lib
    from stkfmm_b200._lib import StkError
    L = lib()
    post, post_wall = L.stk_test_post_wait_error, L.stk_test_post_wall_wait_error
    post.argtypes = [ctypes.c_void_p, ctypes.c_uint]
    post_wall.argtypes = [ctypes.c_void_p, ctypes.c_uint, ctypes.c_int]
    pts, slv, _, td = fmm_case(8, 4000, seed=140)
    f, ref = run_fmm(8, 6, 60, pts, slv, None, td)

    def again():
        out = np.zeros_like(ref)
        f.evaluate_fmm(8, slv, out, None)
        return out

    for look in (again, lambda: f.last_kernel_ms(8)):
        assert post(f.fmm, 8) == 0
        with pytest.raises(StkError):
            look()
        look()
    assert post(f.fmm, 8) == 0
    f.setup_tree(8)
    np.testing.assert_array_equal(again(), ref)

    for kernel, nsub in ((8, 3), (16, 4)):
        pw = pts * [1, 1, 0.45] + [0, 0, 0.01]
        vw = np.concatenate([slv[:, :3], np.full((len(pw), 1), 1e-4)], axis=1)[:, :3 if kernel == 8 else 4]
        w = S.StkWallFMM(6, 60, 0, kernel)
        w.set_box(np.zeros(3), 1.0)
        w.set_points(pw, pw, None)
        w.setup_tree(kernel)

        def wall():
            out = np.zeros((len(pw), 3 if kernel == 8 else 6))
            w.evaluate_fmm(kernel, vw, out)
            return out

        ref_w = wall()
        for look in (wall, w.last_kernel_ms):
            for sub in range(nsub):
                assert post_wall(w.fmm, kernel, sub) == 0
                with pytest.raises(StkError):
                    look()
                look()
        np.testing.assert_array_equal(wall(), ref_w)


@pytest.mark.parametrize("far", [False, True])
def test_evaluations_allocate_no_slots_of_split_sums(torch_cuda, far):
    """A handle evaluated in mixed precision and set to FP64: the slots of its split sums are allocated by
    the switch (near field alone) or the far field's set-up, not by the evaluations that follow."""
    pts, slv, dlv, td = fmm_case(1, 20000, seed=150)
    keep, _ = run_fmm(1, 6, 200, pts, slv, dlv, td)  # libraries and kernels are loaded
    keep.evaluate_near(1, slv, np.zeros((len(pts), td)), dlv)
    f, _ = run_fmm(1, 6, 200, pts, slv, dlv, td, prec=1)

    def evaluate():
        (f.evaluate_fmm if far else f.evaluate_near)(1, slv, np.zeros((len(pts), td)), dlv)

    evaluate()
    before = used_bytes(torch_cuda)
    f.set_precision(0)
    if far:
        evaluate()  # the far field's FP64 set-up
    held = used_bytes(torch_cuda)
    assert held > before, "no split sums in this case"
    evaluate()
    assert used_bytes(torch_cuda) == held
