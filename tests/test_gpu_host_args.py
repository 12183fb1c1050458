"""The native reader of parameter records (csrc/host_args.cpp) against the Python one: the same flat record for
every call it answers for, no answer for any other, and the Python layer's errors in that case."""
import ctypes

import numpy as np
import pytest

import helpers as H
from cumm_b200 import _lib
from cumm_b200 import workloads as W
from cumm_b200.conv.main import ConvMainUnitTest
from cumm_b200.gemm.main import GemmMainUnitTest
from cumm_b200.tensorview import CUDAKernelTimer, float16, from_blob
from cumm_b200.tensorview.gemm import (Activation, ConvOpType, ConvParams, GemmParams, ShuffleStrideType, _conv_args,
                                       _gemm_args, _host)

pytestmark = pytest.mark.gpu


@pytest.fixture
def torch(cuda_lib):
    import torch
    return torch


def native(params):
    """The record the native reader makes, as bytes; None where it leaves the call."""
    conv = isinstance(params, ConvParams)
    args = (_lib.ConvArgs if conv else _lib.GemmArgs)()
    read = _host().conv_args if conv else _host().gemm_args
    return bytes(args) if read(params, ctypes.addressof(args)) else None


def python(params):
    return bytes((_conv_args if isinstance(params, ConvParams) else _gemm_args)(params))


def gemm(torch, shuffle=ShuffleStrideType.ShuffleAC, m=70, k=64, n=72, trans_b=False, with_a_inds=True):
    p = GemmParams()
    p.algo_desp = H.gemm_desp(shuffle, trans_b=trans_b, n=n, k=k)
    half = lambda *s: torch.zeros(s, dtype=torch.float16, device="cuda")
    p.a, p.b, p.c = half(m, k), half(n, k) if trans_b else half(k, n), half(m, n)
    if shuffle == ShuffleStrideType.ShuffleAC:
        i32 = lambda c: torch.arange(c, dtype=torch.int32, device="cuda")
        p.c_inds = i32(33 if with_a_inds else m)
        if with_a_inds:
            p.a_inds = i32(33)
    return p


def conv(torch, op, ksize=(3, 3, 3), C=64, K=72, int8=False):
    tb = W.build_tables(W.sample_coords(300, 5, (8, 24, 24)), grid=(8, 24, 24), ksize=ksize)
    p = ConvParams(3, op)
    p.conv_algo_desp = H.conv_desp(op, C, K, int8_inference=int8)
    p.conv_algo_desp.dynamic_mask = tb.kv > 32
    dt = torch.int8 if int8 else torch.float16
    z = lambda *s, dtype=dt: torch.zeros(s, dtype=dtype, device="cuda")
    p.input, p.weight, p.output = z(tb.n_in, C), z(K, tb.kv, C), z(tb.n_out, K)
    tiles = z((tb.n_out + 127) // 128 * ((tb.kv + 31) // 32), dtype=torch.int32)
    if op == ConvOpType.BackwardInput:
        p.indices, p.mask = H.dev(tb.indices_bwd, torch), H.mask_to_torch(tb.mask_bwd, torch)
        p.mask_argsort = H.dev(tb.mask_argsort_bwd, torch)
    else:
        p.indices, p.mask_argsort = H.dev(tb.indices, torch), H.dev(tb.mask_argsort, torch)
        p.mask = tiles if op == ConvOpType.BackwardWeight else H.mask_to_torch(tb.mask, torch)
        if op == ConvOpType.Forward:
            p.mask_output = tiles
    if op == ConvOpType.BackwardWeight:
        p.mask_width, p.split_k_slices = 128, 32
    if int8:
        p.scale, p.bias = z(K, dtype=torch.float32), z(K, dtype=torch.float32)
    return p


def change(p, **kw):
    for k, v in kw.items():
        setattr(p, k, v)
    return p


def test_same_records(torch):
    zeros = lambda *s, dtype=torch.float16: torch.zeros(s, dtype=dtype, device="cuda")
    plain = ShuffleStrideType.NoShuffle
    calls = [gemm(torch), gemm(torch, trans_b=True), gemm(torch, with_a_inds=False), gemm(torch, plain),
             gemm(torch, plain, trans_b=True),
             change(gemm(torch), a=zeros(70, 128)[:, :64], alpha=0.5, beta=1, act_type=Activation.LeakyReLU, act_alpha=0.25,
                    max_ctas=7)]
    calls += [conv(torch, op, ksize) for ksize in ((3, 3, 3), (5, 5, 5))
              for op in (ConvOpType.Forward, ConvOpType.BackwardInput, ConvOpType.BackwardWeight)]
    s8 = lambda: conv(torch, ConvOpType.Forward, C=64, K=64, int8=True)
    calls += [s8(), change(s8(), output_add=zeros(300, 64, dtype=torch.int8), beta=0.5),
              change(conv(torch, ConvOpType.Forward), bias=zeros(72), beta=1.0, act_type=Activation.ReLU),
              change(conv(torch, ConvOpType.BackwardInput), reverse_mask=True, mask_filter=0x7FFF00FF, max_ctas=3),
              change(conv(torch, ConvOpType.BackwardWeight), weight=zeros(72, 27, 64, dtype=torch.float32))]
    for i, p in enumerate(calls):
        assert native(p) is not None and native(p) == python(p), f"call {i}"


def test_other_calls_are_left_to_the_general_path(torch):
    class Own(ConvParams):
        pass

    zeros = lambda *s, dtype=torch.float16: torch.zeros(s, dtype=dtype, device="cuda")
    fwd = lambda: conv(torch, ConvOpType.Forward)
    unusual = [change(gemm(torch), timer=CUDAKernelTimer(False)), change(gemm(torch), alpha=np.float32(1)),
               change(gemm(torch), d=zeros(72)), change(fwd(), verbose=1), Own(3, ConvOpType.Forward)]
    p = gemm(torch)
    unusual.append(change(p, a=from_blob(p.a.data_ptr(), [70, 64], float16)))
    p = gemm(torch)
    p.algo_desp.trans_c = True
    unusual.append(p)
    for i, p in enumerate(unusual):
        assert native(p) is None, f"unusual call {i}"
    wrong = [(change(gemm(torch), c_inds=None), RuntimeError, "must not empty"),
             (change(gemm(torch), b=zeros(32, 72)), ValueError, "k of a and b"),
             (change(gemm(torch), split_k_slices=2), RuntimeError, "splitk"),
             (change(fwd(), indices=None), RuntimeError, "indices empty"),
             (change(fwd(), mask=zeros(3, dtype=torch.int32)), RuntimeError, "mask has 3 words"),
             (change(fwd(), input=torch.zeros((300, 64), dtype=torch.float16)), RuntimeError, "CUDA device"),
             (change(conv(torch, ConvOpType.BackwardWeight), mask_width=96), RuntimeError, "mask_width")]
    for p, error, text in wrong:
        assert native(p) is None, text
        with pytest.raises(error, match=text):
            (ConvMainUnitTest.implicit_gemm2 if isinstance(p, ConvParams) else GemmMainUnitTest.matmul2)(p)
    # types without a code of the operator surface, in every place where the reader does not look at the type itself
    odd = lambda t: t.new_empty(tuple(t.shape), dtype=torch.complex64)
    for make, names in ((lambda: gemm(torch), ("a_inds", "c_inds")),
                        (lambda: change(fwd(), bias=zeros(72)), ("indices", "mask", "mask_argsort", "mask_output", "bias"))):
        for name in names:
            p = make()
            setattr(p, name, odd(getattr(p, name)))
            assert native(p) is None, name
            with pytest.raises(KeyError):
                (ConvMainUnitTest.implicit_gemm2 if isinstance(p, ConvParams) else GemmMainUnitTest.matmul2)(p)
    # what only the library refuses comes back from the native path as the same error
    p = gemm(torch)
    p.algo_desp.tile_shape = [128, 32, 64]
    with pytest.raises(RuntimeError, match="can't find any suitable algo"):
        GemmMainUnitTest.matmul2(p)
    H.check_status()


def test_same_results_without_the_native_reader(torch, monkeypatch):
    """A layer's calls of both kinds with the extension and without it."""
    import cumm_b200.tensorview.gemm as G
    rng = np.random.default_rng(7)
    fill = lambda t: t.copy_(H.dev(rng.standard_normal(tuple(t.shape)).astype(np.float16), torch))
    calls = [(conv(torch, op), run) for op in (ConvOpType.Forward, ConvOpType.BackwardInput, ConvOpType.BackwardWeight)
             for run in [ConvMainUnitTest.implicit_gemm2]] + [(gemm(torch), GemmMainUnitTest.matmul2)]
    results = []
    for p, run in calls:
        out = p.c if isinstance(p, GemmParams) else (p.output, p.input, p.weight)[int(p.conv_algo_desp.op_type)]
        for t in (p.a, p.b, p.c) if isinstance(p, GemmParams) else (p.input, p.weight, p.output):
            if t is not out:
                fill(t)
        if isinstance(p, ConvParams) and p.conv_algo_desp.op_type == ConvOpType.BackwardWeight:
            p.mask.fill_(0x7FFFFFF)
        run(p)
        results.append((p, run, out, out.clone()))
        assert out.abs().max() > 0
    monkeypatch.setattr(_lib, "load_host", lambda: None)
    monkeypatch.setattr(G, "_HOST", None)
    for p, run, out, want in results:
        out.zero_()
        run(p)
        assert torch.equal(out, want)
    H.check_status()
