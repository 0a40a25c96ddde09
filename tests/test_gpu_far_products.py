"""GPU: the FP64 far field on the int8 tensor cores in whole FMMs: strengths at the ends of the double
range, and the switch between them and cuBLAS."""
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
