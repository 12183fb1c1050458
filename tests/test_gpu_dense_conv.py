"""Dense (non-mask) convolution behind ConvParams (conv_algo_desp.mask_sparse = False), channels
last, against torch.nn.functional.conv{1,2,3}d and its autograd in fp32 on the CPU -- the check
the reference's own dense harness makes (cumm/conv/main_real.py:41-231)."""
import numpy as np
import pytest

import helpers as H
from cumm_b200.conv.main import ConvMainUnitTest
from cumm_b200.tensorview.gemm import ConvOpType, ConvParams

pytestmark = pytest.mark.gpu


def dense_params(op, ndim, C, K, padding, stride, dilation):
    p = ConvParams(ndim, op)
    d = H.conv_desp(op, C, K)
    d.ndim = ndim
    d.mask_sparse = False
    p.conv_algo_desp = d
    p.padding, p.stride, p.dilation = list(padding), list(stride), list(dilation)
    return p


def torch_reference(torch, x, w, dout, padding, stride, dilation):
    """x [N, *S, C], w [K, *k, C], dout [N, *So, K] (numpy fp16) -> out, din, dw in the same layouts (fp32)."""
    import torch.nn.functional as F
    ndim = x.ndim - 2
    to_cf = lambda a: torch.from_numpy(a.astype(np.float32)).movedim(-1, 1).contiguous()
    xt, wt = to_cf(x).requires_grad_(True), to_cf(w).requires_grad_(True)
    conv = {1: F.conv1d, 2: F.conv2d, 3: F.conv3d}[ndim]
    out = conv(xt, wt, None, stride=tuple(stride), padding=tuple(padding), dilation=tuple(dilation))
    din, dw = torch.autograd.grad(out, (xt, wt), to_cf(dout))
    back = lambda t: t.detach().movedim(1, -1).contiguous().numpy()
    return back(out), back(din), back(dw)


@pytest.mark.parametrize("shape,ksize,C,K,padding,stride,dilation", [
    ((2, 6, 10, 12), (3, 3, 3), 32, 48, (1, 1, 1), (1, 1, 1), (1, 1, 1)),
    ((1, 9, 11, 13), (3, 3, 3), 64, 64, (1, 1, 1), (2, 2, 2), (1, 1, 1)),
    ((2, 20, 24), (3, 3), 64, 128, (2, 2), (1, 1), (2, 2)),
    ((3, 200), (5,), 16, 24, (2,), (2,), (1,)),
    ((1, 5, 8, 8), (3, 5, 5), 16, 16, (1, 2, 2), (1, 1, 1), (1, 1, 1)),  # 75 filter offsets: three mask words
])
def test_dense_convolution_against_torch(cuda_lib, shape, ksize, C, K, padding, stride, dilation):
    import torch
    ndim = len(ksize)
    rng = np.random.default_rng(sum(shape) + C)
    x = rng.standard_normal(shape + (C,)).astype(np.float16)
    w = (rng.standard_normal((K,) + ksize + (C,)) / np.sqrt(np.prod(ksize) * C) * 4).astype(np.float16)
    out_sp = tuple((shape[1 + a] + 2 * padding[a] - dilation[a] * (ksize[a] - 1) - 1) // stride[a] + 1 for a in range(ndim))
    dout = rng.standard_normal((shape[0],) + out_sp + (K,)).astype(np.float16)
    want_out, want_din, want_dw = torch_reference(torch, x, w, dout, padding, stride, dilation)
    xd, wd, dd = H.dev(x, torch), H.dev(w, torch), H.dev(dout, torch)
    # forward
    p = dense_params(ConvOpType.Forward, ndim, C, K, padding, stride, dilation)
    out = torch.zeros(dout.shape, dtype=torch.float16, device="cuda")
    p.input, p.weight, p.output = xd, wd, out
    ConvMainUnitTest.implicit_gemm2(p)
    torch.cuda.synchronize()
    H.check_status()
    H.assert_close_f16(out.cpu().numpy(), want_out, "dense forward")
    # backward input
    q = dense_params(ConvOpType.BackwardInput, ndim, C, K, padding, stride, dilation)
    din = torch.zeros(x.shape, dtype=torch.float16, device="cuda")
    q.input, q.weight, q.output = din, wd, dd
    ConvMainUnitTest.implicit_gemm2(q)
    torch.cuda.synchronize()
    H.check_status()
    H.assert_close_f16(din.cpu().numpy(), want_din, "dense backward input")
    # backward weight: sums over all output positions; tolerance grows with their number
    r = dense_params(ConvOpType.BackwardWeight, ndim, C, K, padding, stride, dilation)
    dw = torch.zeros(w.shape, dtype=torch.float16, device="cuda")
    r.input, r.weight, r.output = xd, dw, dd
    r.mask_width = 128
    ConvMainUnitTest.implicit_gemm2(r)
    torch.cuda.synchronize()
    H.check_status()
    got = dw.cpu().numpy().astype(np.float32)
    n_pos = int(np.prod(dout.shape[:-1]))
    tol = H.ATOL * max(1.0, np.sqrt(n_pos) / 64.0) + H.RTOL * np.abs(want_dw)
    assert (np.abs(got - want_dw) <= tol).all(), f"dense backward weight: max abs err {np.abs(got - want_dw).max():.4g}"


def test_dense_convolution_checks_shapes(cuda_lib):
    import torch
    p = dense_params(ConvOpType.Forward, 3, 16, 16, (1, 1, 1), (1, 1, 1), (1, 1, 1))
    p.input = torch.zeros((1, 4, 4, 4, 16), dtype=torch.float16, device="cuda")
    p.weight = torch.zeros((16, 3, 3, 3, 16), dtype=torch.float16, device="cuda")
    p.output = torch.zeros((1, 4, 4, 5, 16), dtype=torch.float16, device="cuda")
    with pytest.raises(RuntimeError, match="output extent"):
        ConvMainUnitTest.implicit_gemm2(p)
    p.output = torch.zeros((64, 16), dtype=torch.float16, device="cuda")
    with pytest.raises(RuntimeError, match="channels-last"):
        ConvMainUnitTest.implicit_gemm2(p)


@pytest.mark.parametrize("shape,ksize,padding,stride,dilation,dtype", [
    ((2, 6, 10, 12), (3, 3, 3), [1, 1, 1], [2, 1, 2], [], "float16"),
    ((1, 20, 24), (3, 3), [2, 2], [], [2, 2], "float32"),
    ((3, 200), (5,), [], [2], [1], "float16"),
    ((1, 5, 8, 8), (3, 5, 5), [1, 2, 2], [1, 1, 1], [1, 1, 1], "float16"),
])
def test_dense_calls_read_in_native_code_are_those_read_in_python(cuda_lib, shape, ksize, padding, stride, dilation, dtype):
    """The second call over a grid is read and launched by the extension: the same results, bit for bit, as the call
    read in Python, with a bias and an activation, with a source of its own, and with an fp32 weight gradient."""
    import torch
    from cumm_b200.dense import _TABLES, run_dense_conv
    from cumm_b200.tensorview.gemm import Activation, _host
    C, K, ndim = 16, 24, len(ksize)
    half = lambda *s: torch.randn(s, device="cuda").half()
    full = lambda v, d: v if v else [d] * ndim
    osp = [(shape[1 + a] + 2 * full(padding, 0)[a] - full(dilation, 1)[a] * (ksize[a] - 1) - 1) // full(stride, 1)[a] + 1
           for a in range(ndim)]
    x, w, dout = half(*shape, C), half(K, *ksize, C), half(shape[0], *osp, K)
    dw = torch.randn((K, *ksize, C), device="cuda").to(getattr(torch, dtype))

    def call(op, host, inp, weight, output, **more):
        p = dense_params(op, ndim, C, K, padding, stride, dilation)
        p.input, p.weight, p.output = inp, weight, output
        for k, v in more.items():
            setattr(p, k, v)
        run_dense_conv(p, host)
        torch.cuda.synchronize()
        return p

    F, D, W = ConvOpType.Forward, ConvOpType.BackwardInput, ConvOpType.BackwardWeight
    bias = half(K)
    for op, out, more in ((F, "out", dict(bias=bias, beta=1.0, act_type=Activation.ReLU)), (F, "out", dict(alpha=0.5, beta=2.0)),
                          (D, "in", {}), (W, "w", {}), (W, "w", dict(beta=0.5))):
        made = []
        for host in (None, _host()):
            t = {"in": x.clone(), "w": dw.clone() if op == W else w, "out": dout.clone()}
            p = call(op, host, t["in"], t["w"], t["out"], **more)
            made.append(t[out])
        assert torch.equal(*made), (op, more)
        # and it was the extension that answered
        import ctypes
        from cumm_b200 import _lib
        tables = _TABLES[_host().dense_key(p)]["native"]
        assert _host().run_dense(p, tables, ctypes.addressof(_lib.ConvArgs())) == (True if op == W else 0)
    # what it leaves to Python: lists of the wrong length, an output that does not fit
    for field, value in (("padding", [1] * (ndim + 1)), ("output", dout[..., :8].contiguous())):
        p = dense_params(F, ndim, C, K, padding, stride, dilation)
        p.input, p.weight, p.output = x, w, dout
        setattr(p, field, value)
        with pytest.raises(RuntimeError):
            run_dense_conv(p, _host())
    torch.cuda.synchronize()
    H.check_status()


@pytest.mark.parametrize("first", ["on a busy stream", "captured"])
def test_the_first_call_over_a_grid_makes_whole_tables(cuda_lib, first):
    """The first call over a grid on a stream other than torch's, directly followed by calls on another one, while torch's
    own stream is busy; and captured, with eager calls before the graph has run.  All three operators, against
    the same calls with everything in between waited for, bit for bit."""
    import torch
    from cumm_b200.dense import _TABLES
    shape, ksize, C, K = (2, 37, 45), (3, 3), 32, 48
    half = lambda *s: torch.randn(s, device="cuda").half()
    x, w, dout = half(*shape, C), half(K, *ksize, C), half(*shape, K)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]

    def results():
        return {ConvOpType.Forward: torch.zeros_like(dout), ConvOpType.BackwardInput: torch.zeros_like(x),
                ConvOpType.BackwardWeight: torch.zeros_like(w)}

    def call(op, made, stream):
        p = dense_params(op, 2, C, K, (1, 1), (1, 1), (1, 1))
        t = {ConvOpType.Forward: dout, ConvOpType.BackwardInput: x, ConvOpType.BackwardWeight: w}
        t[op] = made[op]
        p.input, p.weight, p.output = t[ConvOpType.BackwardInput], t[ConvOpType.BackwardWeight], t[ConvOpType.Forward]
        p.stream, p.mask_width = stream.cuda_stream, 128
        ConvMainUnitTest.implicit_gemm2(p)

    want, made, eager = results(), results(), results()
    for i, op in enumerate(want):  # the library's and torch's scratch is there before anything is captured
        call(op, want, torch.cuda.default_stream())
        call(op, want, streams[0])
        torch.cuda.synchronize()
    want = {op: t.clone() for op, t in want.items()}
    big = half(4096, 4096)
    torch.cuda.synchronize()
    _TABLES.clear()
    if first == "captured":
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=streams[0]):
            for op in made:
                call(op, made, streams[0])
        for op in eager:
            call(op, eager, streams[1])
        streams[1].synchronize()
        g.replay()
    else:
        for _ in range(20):
            big @ big
        for op in made:
            call(op, made, streams[0])
            call(op, eager, streams[1])
    torch.cuda.synchronize()
    H.check_status()
    for op in want:
        assert torch.equal(made[op], want[op]) and torch.equal(eager[op], want[op]), op
