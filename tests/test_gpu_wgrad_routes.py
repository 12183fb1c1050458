"""The weight gradient's routes -- row lists or row tiles per offset, stage layouts by channel
counts -- and the forward / input-gradient items of outputs wider than a tile, at the edges of each."""
import numpy as np
import pytest

import helpers as H
from cumm_b200 import workloads as W
from cumm_b200.layer import DeviceTables, SparseConvLayer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch(cuda_lib):
    import torch
    return torch


def operands(tb, C, K, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((tb.n_in, C)).astype(np.float16)
    dout = rng.standard_normal((tb.n_out, K)).astype(np.float16)
    w = (rng.standard_normal((K, tb.kv, C)) / np.sqrt(tb.kv * C) * 4).astype(np.float16)
    return x, dout, w


# (rows, grid), all of up to 64 tiles, whose lists one launch makes and which always have room: nothing but
# the centre; one row past a tile; half full (most offsets listed); three fifths full; solid (nothing listed)
SCENES = [(1, (8, 24, 24)), (129, (8, 24, 24)), (2300, (8, 24, 24)), (2900, (8, 24, 24)), (4608, (8, 24, 24))]


@pytest.mark.parametrize("C,K", [(64, 64), (32, 72), (128, 64), (64, 128), (200, 136)])
@pytest.mark.parametrize("n,grid", SCENES)
def test_weight_gradient_by_rows(torch, oracle, n, grid, C, K):
    tb = W.build_tables(W.sample_coords(n, 60 + n, grid), grid=grid)
    x, dout, _ = operands(tb, C, K, n)
    tiles = np.bitwise_or.reduceat(tb.mask, np.arange(0, n, 128))
    got = H.run_conv_wgrad(torch, dout, x, tb, tiles)  # scratch from the library: lists
    H.check_status()
    want = oracle.mask_igemm_wgrad(dout, x, np.zeros((K, 27, C), np.float16), tb.indices, tiles, tb.mask_argsort)
    H.assert_close_wgrad(got, want, tb.indices, f"n={n} C={C} K={K}")


@pytest.mark.parametrize("ksize,n,grid,mask_width,mask_filter", [
    # three fifths full: more listed pairs than there is room for, the last offsets are walked by tiles
    ((3, 3, 3), 33500, (16, 60, 60), 128, 0xFFFFFFFF), ((3, 3, 3), 33500, (16, 60, 60), 32, 0xFFFFFFFF),
    ((3, 3, 3), 33500, (16, 60, 60), 256, 0xFFFFFFFF), ((3, 3, 3), 33500, (16, 60, 60), 128, 0x5A5A5A5),
    # a few rows per offset beside a full centre; the centre filtered out; nothing left
    ((3, 3, 3), 32769, (41, 300, 300), 128, 0xFFFFFFFF), ((3, 3, 3), 40000, (41, 300, 300), 64, ~(1 << 13)),
    ((3, 3, 3), 32769, (41, 300, 300), 128, 0),
    # around the line between one launch and two, and the last size whose lists have room for all rows
    ((3, 3, 3), 8192, (16, 30, 30), 128, 0xFFFFFFFF), ((3, 3, 3), 8193, (16, 30, 30), 128, 0xFFFFFFFF),
    ((3, 3, 3), 32768, (16, 59, 59), 128, 0xFFFFFFFF), ((5, 5, 5), 32768, (20, 120, 120), 128, 0xFFFFFFFF),
    # four mask words: all listed, and too many
    ((5, 5, 5), 33000, (20, 120, 120), 128, 0xFFFFFFFF), ((5, 5, 5), 33000, (16, 80, 80), 128, 0xFFFFFFFF)])
def test_row_lists_in_two_launches(torch, ksize, n, grid, mask_width, mask_filter):
    """Plans made by two kernels, and the last sizes that one makes.  Integers sum exactly: lists and tiles
    give the same bits."""
    tb = W.build_tables(W.sample_coords(n, 5, grid), grid=grid, ksize=ksize)
    per_row = tb.num_pairs / n - 1
    room = 8 + tb.kv // 8
    if grid in ((16, 60, 60), (16, 80, 80)):
        assert per_row > room, "the lists do not overflow"
    rng = np.random.default_rng(n)
    x = rng.integers(-2, 3, (n, 32)).astype(np.float16)
    dout = rng.integers(-2, 3, (n, 40)).astype(np.float16)
    masks = np.bitwise_or.reduceat(tb.mask, np.arange(0, n, mask_width), axis=0)
    flt = mask_filter & 0xFFFFFFFF
    by = [H.run_conv_wgrad(torch, dout, x, tb, masks, kv=tb.kv, mask_width=mask_width, mask_filter=flt, fp32_out=True,
                           row_lists=lists) for lists in (True, False)]
    H.check_status()
    want = np.zeros((40, tb.kv, 32))
    xs, ds = torch.from_numpy(x).cuda().double(), torch.from_numpy(dout).cuda().double()
    for f in range(tb.kv):
        if (flt >> (f % 32)) & 1:
            o = np.flatnonzero(tb.indices[f] >= 0)
            i = torch.from_numpy(tb.indices[f][o].astype(np.int64)).cuda()
            want[:, f] = (ds[torch.from_numpy(o).cuda()].T @ xs[i]).cpu().numpy()
    assert (by[0] == want).all() and (by[1] == want).all()


def test_weight_gradient_in_scratch_of_either_size(torch):
    """A buffer of the caller's that holds tile lists only is walked by tiles; integers sum exactly, so
    both ways give the same bits, and so does a prepared layer, planned once, at every launch."""
    from cumm_b200.conv.main import ConvMainUnitTest
    from cumm_b200.layer import make_desp
    from cumm_b200.tensorview.gemm import ConvOpType, ConvParams, _conv_args
    from cumm_b200 import _lib
    import ctypes
    grid, n, C, K = (8, 24, 24), 2900, 64, 96
    t = DeviceTables.from_host(W.build_tables(W.sample_coords(n, 3, grid), grid=grid), "cuda")
    g = torch.Generator().manual_seed(4)
    x = torch.randint(-2, 3, (n, C), generator=g).half().cuda()
    dout = torch.randint(-2, 3, (n, K), generator=g).half().cuda()
    results = []
    for size_of in (_lib.load().cb2_conv_workspace_size, _lib.load().cb2_conv_workspace_size_lists):
        dw = torch.zeros((K, 27, C), dtype=torch.float32, device="cuda")
        p = ConvParams(3, ConvOpType.BackwardWeight)
        p.conv_algo_desp = make_desp(ConvOpType.BackwardWeight, False, C, K)
        p.input, p.weight, p.output = x, dw, dout
        p.indices, p.mask, p.mask_argsort = t.indices, t.mask_output, t.mask_argsort
        p.mask_width, p.split_k_slices = 128, 32
        p.workspace = torch.empty(size_of(ctypes.byref(_conv_args(p))) + 256, dtype=torch.uint8, device="cuda")
        ConvMainUnitTest.implicit_gemm2(p)
        results.append(dw)
    dw = torch.zeros_like(results[0])
    layer = SparseConvLayer(t, torch.zeros((K, 27, C), dtype=torch.float16, device="cuda"), x,
                            torch.zeros((n, K), dtype=torch.float16, device="cuda"), dout, torch.zeros_like(x), dw)
    for _ in range(3):
        dw.zero_()
        layer.wgrad.launch()
        torch.cuda.synchronize()
        H.check_status()
        assert torch.equal(dw, results[0])
    assert torch.equal(results[0], results[1])
    # a plan is reused as what it is: tiles then lists allowed, and the other way round; made in a record of
    # the smaller size and used in one of the larger, and the other way round
    lists = _lib.CB2_PLAN_ROW_LISTS
    large, small = p.workspace.numel(), _lib.load().cb2_conv_workspace_size(ctypes.byref(_conv_args(p)))
    for steps in (((0, large), (1 | lists, large)), ((lists, large), (1, large)),
                  ((lists, small), (1 | lists, large)), ((lists, large), (1 | lists, small))):
        args = _conv_args(p)
        p.workspace.fill_(0x7f)  # nothing left of an earlier plan
        args.workspace = p.workspace.data_ptr()
        for args.reuse_plan, args.workspace_bytes in steps:
            p.weight.zero_()
            _lib.raise_for(_lib.load().cb2_conv_run(ctypes.byref(args), None))
            torch.cuda.synchronize()
            H.check_status()
            assert torch.equal(p.weight, dw)
    want = torch.zeros((27, K, C), dtype=torch.float64)
    for f in range(27):
        o = torch.nonzero(t.indices[f] >= 0).flatten().cpu()
        want[f] = dout.cpu().double()[o].T @ x.cpu().double()[t.indices[f].cpu()[o].long()]
    assert torch.equal(results[0].cpu().double(), want.permute(1, 0, 2))


@pytest.mark.parametrize("n", [127, 2300])
@pytest.mark.parametrize("C,K", [(64, 136), (136, 64), (192, 384), (256, 264)])
def test_outputs_wider_than_a_tile(torch, oracle, n, C, K):
    """Column parts drawn with the tiles: a last part of eight columns, three parts, kernels that
    reduce in one pass and in several; tile masks written once."""
    tb = W.build_tables(W.sample_coords(n, 70 + n, (8, 24, 24)), grid=(8, 24, 24))
    x, dout, w = operands(tb, C, K, n + 1)
    got, mo = H.run_conv_fwd(torch, x, w, tb)
    H.check_status()
    mo_ref = np.zeros_like(mo)
    want = oracle.mask_igemm(x, w, np.zeros((n, K), np.float16), tb.indices, tb.mask, tb.mask_argsort, mask_out=mo_ref)
    assert (mo == mo_ref).all()
    H.assert_close_f16(got, want, f"forward n={n} C={C} K={K}")
    din = H.run_conv_dgrad(torch, dout, w, tb)
    H.check_status()
    H.assert_close_f16(din, oracle.mask_igemm(dout, w, np.zeros((n, C), np.float16), tb.indices_bwd, tb.mask_bwd,
                                              tb.mask_argsort_bwd, is_dgrad=True), f"dgrad n={n} C={C} K={K}")
