"""GPU: sums whose sources are split over warps (direct sums in chunks, list items in parts), and
FP64 FMMs with their products on the int8 tensor cores against the same FMMs on cuBLAS.

Sums: 1e-12 relative L2 of the oracle (FP64 pair sums of a few thousand terms: 2^-53 sqrt(n) and a
few roundings a pair), 1e-6 mixed, as for every other list; the parts are added in a fixed order, so
that a repeat gives the same bits."""
import numpy as np
import pytest

from conftest import rel_l2
from helpers import UK_TDIM, uk_values
from oracle import oracle as O
from test_gpu_direct import gpu_direct
from test_gpu_fmm import fmm_case, run_fmm
from test_gpu_lists import dev, oracle_ulist, run_lists

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return torch


# one source tile and its edges, one target slot and its edges, a few targets with very many chunks
@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 1e-6)])
@pytest.mark.parametrize("ns,nt", [(31, 2), (32, 17), (33, 33), (4099, 64), (4099, 65), (40000, 1), (20001, 129)])
@pytest.mark.parametrize("uk", [6, 10])
def test_direct_chunks(torch_cuda, uk, ns, nt, prec, tol):
    from stkfmm_b200 import lib
    rng = np.random.default_rng(ns + nt)
    src, val, trg = rng.random((ns, 3)), uk_values(rng, uk, ns), rng.random((nt, 3))
    trg[0] = src[0]
    start = rng.normal(size=(nt, UK_TDIM[uk]))
    a = gpu_direct(torch_cuda, lib(), uk, src, val, trg, prec, out0=start)
    assert rel_l2(a - start, O.direct(uk, src, val, trg)) < tol
    if prec == 0:
        np.testing.assert_array_equal(a, gpu_direct(torch_cuda, lib(), uk, src, val, trg, prec, out0=start))


def long_lists(uk, seed):
    """Target boxes of 1 to 200 targets; lists with empty boxes first, last and between, boxes of one
    source, boxes that several parts cut, images; one box without targets, one without a list."""
    rng = np.random.default_rng(seed)
    size = [0, 1, 700, 0, 3, 2500, 33, 0, 64, 4000, 1, 0]
    sb = np.concatenate([[0], np.cumsum(size)[:-1]])
    se = sb + size
    src = rng.random((sum(size), 3))
    nts = [1, 200, 0, 65, 9, 30]
    tb = np.concatenate([[0], np.cumsum(nts)[:-1]])
    te = tb + nts
    lists = [list(range(12)), [0, 9, 9, 5, 3], [2], [], [5, 11, 2, 0], [11, 1, 10]]
    code = [[int(rng.integers(0, 27)) if i else 13 for i in range(len(x))] for x in lists]
    off = np.concatenate([[0], np.cumsum([len(x) for x in lists])])
    ent = np.array([b << 5 | c for x, cc in zip(lists, code) for b, c in zip(x, cc)], np.int32)
    trg = rng.random((sum(nts), 3))
    trg[1:20] = src[200:219]  # coincident pairs
    return tb, te, off, ent, sb, se, src, uk_values(rng, uk, len(src)), trg


@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 1e-6)])
@pytest.mark.parametrize("uk", [1, 4, 20])
def test_lists_in_parts(torch_cuda, uk, prec, tol):
    case = long_lists(uk, 5 + uk)
    a = run_lists(torch_cuda, uk, prec, *case)
    assert rel_l2(a, oracle_ulist(uk, *case)) < tol
    np.testing.assert_array_equal(a, run_lists(torch_cuda, uk, prec, *case))


@pytest.mark.parametrize("uk", [4, 20])  # 3 and 16 components: both of the plan's buffers
def test_plan_parts_first_met_in_a_capture(torch_cuda, uk):
    """A plan warmed up in mixed precision and captured in FP64, whose split sums then need their
    buffer: the replay gives what an execution outside gives."""
    from stkfmm_b200 import lib
    from stkfmm_b200._lib import P_i, check
    torch, L = torch_cuda, lib()
    tb, te, off, ent, sb, se, src, val, trg = long_lists(uk, 9)
    arrs = [np.ascontiguousarray(x, dtype=np.int32) for x in (tb, te, off, ent, sb, se)]
    p = [a.ctypes.data_as(P_i) for a in arrs]
    plan = L.stk_p2p_plan_create(len(tb), p[0], p[1], p[2], p[3], len(sb), p[4], p[5], len(src), len(trg), 1.0, None)
    assert plan
    try:
        s, v, t = dev(torch, src), dev(torch, val), dev(torch, trg)
        out = torch.zeros((len(trg), UK_TDIM[uk]), dtype=torch.float64, device="cuda")

        def execute(prec):
            check(L.stk_p2p_plan_execute(plan, uk, prec, s.data_ptr(), v.data_ptr(), t.data_ptr(), None, out.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream), "plan")

        execute(1)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            execute(0)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        out.zero_()
        execute(0)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(got, out.cpu().numpy())
        assert rel_l2(got, oracle_ulist(uk, tb, te, off, ent, sb, se, src, val, trg)) < 1e-12
        del graph
    finally:
        torch.cuda.synchronize()
        L.stk_p2p_plan_destroy(plan)


# LapPGrad with few chunks, Stokes, RPY (scaled, 4 densities), PVel; p whose surfaces are no multiple of 32
@pytest.mark.parametrize("kernel,p,max_pts", [(1, 10, 60), (2, 7, 60), (16, 8, 60), (128, 6, 150)])
def test_fp64_fmm_int8_products(torch_cuda, monkeypatch, kernel, p, max_pts):
    """The noise of an FMM: values three times as large, rounded differently throughout, give three
    times the result but for it.  The int8 products' may not be above cuBLAS's, and the two paths
    differ by it (each within a factor for the two draws, plus the near field's 1e-14)."""
    pts, slv, dlv, td = fmm_case(kernel, 9000, seed=60 + kernel)
    lin = slice(0, 3) if kernel == 16 else slice(None)  # RPY's fourth value is a radius
    slv3 = slv.copy()
    slv3[:, lin] *= 3.0
    res, noise = {}, {}
    for mode in ("0", "1"):
        monkeypatch.setenv("STKFMM_F64_I8", mode)
        _, res[mode] = run_fmm(kernel, p, max_pts, pts, slv, dlv, td)
        _, r3 = run_fmm(kernel, p, max_pts, pts, slv3, None if dlv is None else 3.0 * dlv, td)
        noise[mode] = rel_l2(r3 / 3.0, res[mode])
    assert noise["1"] < 2.0 * noise["0"] + 1e-14, noise
    assert rel_l2(res["1"], res["0"]) < 4.0 * noise["0"] + 1e-14, (rel_l2(res["1"], res["0"]), noise)


@pytest.mark.parametrize("kernel,max_pts", [(2, 40), (16, 60), (128, 60)])
def test_mixed_fmm_keeps_its_fp64_products(torch_cuda, monkeypatch, kernel, max_pts):
    """The mixed path of the Stokes translations rounds to FP32 after its FP64 products and stays with
    cuBLAS for them: the same numbers with the int8 products on and off (a rebuilt operator set, 1e-13
    as for any two handles that built their own)."""
    pts, slv, dlv, td = fmm_case(kernel, 9000, seed=80 + kernel)
    res = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("STKFMM_F64_I8", mode)
        _, res[mode] = run_fmm(kernel, 8, max_pts, pts, slv, dlv, td, prec=1)
    assert rel_l2(res["1"], res["0"]) < 1e-13
