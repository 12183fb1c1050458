"""Launches that overlap on the GPU: a captured forward replayed on one stream while eager
forwards loop on another, and one prepared call launched back to back.  Every prepared call
owns its tile-ticket counters, so two calls never draw tiles from the same counter, whatever
the library's round-robin pool hands to other launches in between; results are checked against
the oracle."""
import numpy as np
import pytest

import helpers as H
from cumm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_graph_replay_beside_eager_launches(cuda_lib, oracle):
    import torch
    from cumm_b200.layer import DeviceTables, SparseConvLayer
    grid = (8, 48, 48)
    C = K = 64
    layers, wants, outs = [], [], []
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for i, n in enumerate((9000, 7000)):
        tb = W.build_tables(W.sample_coords(n, 700 + i, grid), grid=grid)
        rng = np.random.default_rng(710 + i)
        x = rng.standard_normal((tb.n_in, C)).astype(np.float16)
        w = (rng.standard_normal((K, 27, C)) / 16).astype(np.float16)
        out = torch.zeros((tb.n_out, K), dtype=torch.float16, device="cuda")
        with torch.cuda.stream(streams[i]):
            layers.append(SparseConvLayer(DeviceTables.from_host(tb, "cuda"), H.dev(w, torch), H.dev(x, torch), out,
                                          stream=streams[i].cuda_stream))
        outs.append(out)
        wants.append(oracle.mask_igemm(x, w, np.zeros((tb.n_out, K), np.float16), tb.indices, tb.mask, tb.mask_argsort))
    torch.cuda.synchronize()
    a, b = layers
    with torch.cuda.stream(streams[0]):
        a.fwd.launch()
        streams[0].synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=streams[0]):
            for _ in range(4):
                a.fwd.launch()
    for rounds in range(20):
        with torch.cuda.stream(streams[0]):
            g.replay()
        with torch.cuda.stream(streams[1]):
            for _ in range(6):
                b.fwd.launch()
        if rounds % 5 == 4:
            # launches of other calls in between advance the library's own pool of counters
            with torch.cuda.stream(streams[1]):
                H.run_conv_fwd(torch, np.zeros((8, C), np.float16), np.zeros((K, 27, C), np.float16),
                               W.build_tables(W.sample_coords(8, 1, grid), grid=grid))
    torch.cuda.synchronize()
    H.check_status()
    H.assert_close_f16(outs[0].cpu().numpy(), wants[0], "captured forward replayed beside eager launches")
    H.assert_close_f16(outs[1].cpu().numpy(), wants[1], "eager forward beside graph replays")


def test_the_same_prepared_call_back_to_back(cuda_lib, oracle):
    """One prepared int8 forward launched many times in a row on one stream, eagerly and from a
    graph: int8 convolutions are launched with programmatic dependent launch, so a launch starts
    drawing tiles while its predecessor -- the same call -- still runs.  The call alternates
    between two pairs of ticket counters; every launch must leave the bit-exact result."""
    import torch
    from cumm_b200.layer import DeviceTables, SparseConvLayer
    grid = (8, 64, 64)
    C = K = 128
    tb = W.build_tables(W.sample_coords(20000, 721, grid), grid=grid, stride=(2, 2, 2), subm=False)
    rng = np.random.default_rng(722)
    x = rng.integers(-127, 128, (tb.n_in, C)).astype(np.int8)
    w = rng.integers(-127, 128, (K, 27, C)).astype(np.int8)
    scale = rng.uniform(1e-3, 1e-2, K).astype(np.float32)
    bias = rng.standard_normal(K).astype(np.float32)
    want = oracle.mask_igemm_s8(x, w, np.zeros((tb.n_out, K), np.int8), scale, bias, tb.indices, tb.mask,
                                tb.mask_argsort)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        out = torch.zeros((tb.n_out, K), dtype=torch.int8, device="cuda")
        L = SparseConvLayer(DeviceTables.from_host(tb, "cuda"), H.dev(w, torch), H.dev(x, torch), out,
                            stream=stream.cuda_stream)
        L.prepare_int8(H.dev(scale, torch), H.dev(bias, torch))
        for _ in range(7):
            L.fwd.launch()
        stream.synchronize()
        H.check_status()
        assert (out.cpu().numpy() == want).all(), "eager launches back to back"
        out.zero_()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            for _ in range(5):
                L.fwd.launch()
        for _ in range(3):
            g.replay()
        stream.synchronize()
    H.check_status()
    assert (out.cpu().numpy() == want).all(), "graph of back-to-back launches, replayed"


def _small_scenes(oracle, channels, count, n=2000, grid=(8, 24, 24)):
    """Scenes of one row count, weights for a layer per step of ``channels``, and what the layers make of them."""
    rng = np.random.default_rng(731)
    ws = [(rng.standard_normal((K, 27, C)) / np.sqrt(27 * C)).astype(np.float16) for C, K in zip(channels, channels[1:])]
    scenes = []
    for i in range(count):
        coords = W.sample_coords(n, 730 + i, grid)
        tb = W.build_tables(coords, grid=grid)
        x = rng.standard_normal((n, channels[0])).astype(np.float16)
        want = [x]
        for w in ws:
            want.append(oracle.mask_igemm(want[-1], w, np.zeros((n, w.shape[0]), np.float16), tb.indices, tb.mask,
                                          tb.mask_argsort))
        scenes.append((coords, tb, x, want[1:]))
    return ws, scenes


def _forward(p, x, w, out, indices, mask, argsort, stream=0):
    from cumm_b200.conv.main import ConvMainUnitTest
    p.input, p.weight, p.output = x, w, out
    p.indices, p.mask, p.mask_argsort, p.stream = indices, mask, argsort, stream
    ConvMainUnitTest.implicit_gemm2(p)


def _params(ws):
    from cumm_b200.tensorview.gemm import ConvOpType, ConvParams
    ps = []
    for w in ws:
        p = ConvParams(3, ConvOpType.Forward)
        p.conv_algo_desp = H.conv_desp(ConvOpType.Forward, w.shape[2], w.shape[0])
        ps.append(p)
    return ps


def test_small_layers_directly_behind_their_table_build(cuda_lib, oracle):
    """Tables of one scene after the other, and layer into layer of each, on one stream without a synchronisation: the
    tables of the next scene come to lie where the last one's were, activations are overwritten.  The launches
    are those that clusters share, which start under their predecessor's end."""
    import torch
    from cumm_b200.pairgen import build_tables_gpu
    grid = (8, 24, 24)
    ws, scenes = _small_scenes(oracle, (64, 64, 128, 48), 6)
    wd, ps = [H.dev(w, torch) for w in ws], _params(ws)
    coords, xs = [H.dev(s[0], torch) for s in scenes], [H.dev(s[2], torch) for s in scenes]
    acts = [torch.zeros((2000, w.shape[0]), dtype=torch.float16, device="cuda") for w in ws]
    outs = []
    torch.cuda.synchronize()
    for rounds in range(5):
        for i in range(len(scenes)):
            t = build_tables_gpu(coords[i], 1, grid)
            h = xs[i]
            for p, w, act in zip(ps, wd, acts):
                _forward(p, h, w, act, t.indices, t.mask, t.mask_argsort)
                h = act
            outs.append((i, [a.clone() for a in acts]))
    torch.cuda.synchronize()
    H.check_status()
    for k, (i, got) in enumerate(outs):
        for layer, (g, want) in enumerate(zip(got, scenes[i][3])):
            H.assert_close_f16(g.cpu().numpy(), want, f"pass {k}, scene {i}, layer {layer}")


def test_small_layers_captured_behind_the_kernels_that_write_their_tables(cuda_lib, oracle):
    """The same as a graph: kernels write the tables in place, the layers follow at once; replayed on other tables."""
    import torch
    ws, scenes = _small_scenes(oracle, (64, 64, 128), 4)
    wd, ps = [H.dev(w, torch) for w in ws], _params(ws)
    hold = lambda tb: [H.dev(tb.indices, torch), H.mask_to_torch(tb.mask, torch), H.dev(tb.mask_argsort, torch)]
    src, here = hold(scenes[0][1]), hold(scenes[0][1])
    x = H.dev(scenes[0][2], torch)
    acts = [torch.zeros((2000, w.shape[0]), dtype=torch.float16, device="cuda") for w in ws]
    stream = torch.cuda.Stream()

    def step():
        h = x
        for p, w, act in zip(ps, wd, acts):
            for a, b in zip(src, here):
                torch.add(a, 0, out=b)
            _forward(p, h, w, act, *here, stream=stream.cuda_stream)
            h = act

    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        step()
        stream.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            step()
            step()
        for rounds in range(12):
            _, tb, feats, want = scenes[rounds % 4]
            for a, b in zip(src, hold(tb)):
                a.copy_(b)
            x.copy_(H.dev(feats, torch))
            g.replay()
            g.replay()
            got = [a.cpu().numpy() for a in acts]
            for layer in range(len(ws)):
                H.assert_close_f16(got[layer], want[layer], f"replay {rounds}, layer {layer}")
    H.check_status()


def test_every_launch_of_a_chain_does_its_work_once(cuda_lib):
    """One record launched many times in a row, each launch adding one to every output in place: a tile that a launch
    leaves out or does twice stays visible.  Launches of fewer tiles than SMs, some of many offsets and most of one, so
    that a launch's successors find SMs free while its heaviest tiles still run."""
    import torch
    from cumm_b200.layer import make_desp
    from cumm_b200.tensorview.gemm import ConvOpType, ConvParams, GemmParams, ShuffleStrideType, prepare_conv, prepare_gemm
    side = np.arange(17, dtype=np.int32)
    block = np.stack(np.meshgrid([0], side + 3, side + 9, side + 9, indexing="ij"), -1).reshape(-1, 4)
    sparse = W.sample_coords(5000, 741, (41, 300, 300))
    coords = np.unique(np.concatenate([block, sparse]), axis=0).astype(np.int32)
    tb = W.build_tables(np.random.default_rng(742).permutation(coords), grid=(41, 300, 300))
    n, C, launches = tb.n_out, 128, 100
    assert 128 * 70 < n < 128 * 80
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        out = torch.zeros((n, C), dtype=torch.int8, device="cuda")
        p = ConvParams(3, ConvOpType.Forward)
        p.conv_algo_desp = make_desp(ConvOpType.Forward, True, C, C)
        p.input = torch.ones((n, C), dtype=torch.int8, device="cuda")
        p.weight = torch.ones((C, 27, C), dtype=torch.int8, device="cuda")
        p.output = p.output_add = out
        p.scale, p.bias = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
        p.beta, p.stream = 1.0, stream.cuda_stream
        p.indices, p.mask, p.mask_argsort = H.dev(tb.indices, torch), H.mask_to_torch(tb.mask, torch), H.dev(tb.mask_argsort, torch)
        a = torch.zeros((n, 64), dtype=torch.float16, device="cuda")
        a[:, 0] = 1
        q = GemmParams()
        q.algo_desp = H.gemm_desp(ShuffleStrideType.ShuffleAC, trans_b=True, n=64, k=64)
        q.a, q.b, q.c = a, torch.ones((64, 64), dtype=torch.float16, device="cuda"), torch.zeros_like(a)
        q.a_inds = q.c_inds = torch.randperm(n, device="cuda").int()
        q.beta, q.stream = 1.0, stream.cuda_stream
        stream.synchronize()
        for call, dst in ((prepare_conv(p), out), (prepare_gemm(q), q.c)):
            for _ in range(launches):
                call.launch()
            stream.synchronize()
            assert bool((dst == launches).all()), "eager launches"
            dst.zero_()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                for _ in range(launches // 4):
                    call.launch()
            for _ in range(4):
                g.replay()
            stream.synchronize()
            assert bool((dst == launches).all()), "captured launches"
    H.check_status()


@pytest.mark.parametrize("n,grid,C", [(2000, (8, 24, 24), 64), (9000, (8, 48, 48), 128), (30011, (12, 80, 80), 32)])
def test_layers_that_read_what_their_predecessor_writes(cuda_lib, n, grid, C):
    """Two prepared layers over fixed tables, forward and backward, each launch reading what the one before it wrote:
    from the second round on they read their tables and plans while that one still runs.  Input rows change every
    round; results are those of calls with everything in between waited for, bit for bit."""
    import torch
    from cumm_b200.layer import DeviceTables, SparseConvLayer
    rng = np.random.default_rng(741)
    t = DeviceTables.from_host(W.build_tables(W.sample_coords(n, 740, grid), grid=grid), "cuda")
    half = lambda *shape: H.dev((rng.standard_normal(shape) / 8).astype(np.float16), torch)
    rows, grads = [half(n, C) for _ in range(4)], [half(n, C) for _ in range(4)]
    ws = [half(C, t.kv, C), half(C, t.kv, C)]

    def layers(stream):
        b = {k: torch.zeros((n, C), dtype=torch.float16, device="cuda") for k in ("x", "y", "z", "dz", "dy", "dx")}
        b.update({k: torch.zeros((C, t.kv, C), dtype=torch.float16, device="cuda") for k in ("dw1", "dw2")})
        one = SparseConvLayer(t, ws[0], b["x"], b["y"], b["dy"], b["dx"], b["dw1"], stream=stream.cuda_stream)
        two = SparseConvLayer(t, ws[1], b["y"], b["z"], b["dz"], b["dy"], b["dw2"], stream=stream.cuda_stream)
        return b, [one.fwd, two.fwd, two.dgrad, two.wgrad, one.wgrad, one.dgrad]

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        want_b, alone = layers(stream)
        b, calls = layers(stream)
        for i in range(4):
            for buf in (want_b, b):
                buf["x"].copy_(rows[i])
                buf["dz"].copy_(grads[i])
            for c in alone:
                stream.synchronize()
                c.launch()
            stream.synchronize()
            if i < 2:
                for c in calls:
                    c.launch()
            else:  # captured, the round twice over
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=stream):
                    for c in calls + calls:
                        c.launch()
                g.replay()
            stream.synchronize()
            H.check_status()
            for k, v in want_b.items():
                assert torch.equal(v, b[k]), (i, k)


@pytest.mark.parametrize("n,grid,C", [(30011, (12, 80, 80), 64), (20000, (12, 64, 64), 72), (9000, (8, 48, 48), 128)])
def test_layers_directly_behind_new_tables_in_old_places(cuda_lib, n, grid, C):
    """Calls that do not say their tables are as they were, each directly behind whatever wrote its tables, masks and rows
    into the buffers that the call before it still reads (gather4, cp.async, one tile a CTA): forward and input gradient
    of scene after scene are those of calls with everything in between waited for, bit for bit."""
    import torch
    from cumm_b200.conv.main import ConvMainUnitTest
    from cumm_b200.layer import DeviceTables
    from cumm_b200.tensorview.gemm import ConvOpType, ConvParams
    rng = np.random.default_rng(751)
    scenes = [DeviceTables.from_host(W.build_tables(W.sample_coords(n, 750 + i, grid), grid=grid), "cuda") for i in range(3)]
    half = lambda *shape: H.dev((rng.standard_normal(shape) / 8).astype(np.float16), torch)
    rows, w = [half(n, C) for _ in scenes], half(C, 27, C)
    names = ("indices", "mask", "mask_argsort", "indices_bwd", "mask_bwd", "mask_argsort_bwd")
    here = scenes[0].clone()
    x = torch.zeros_like(rows[0])

    def call(op, inp, out, stream):
        p = ConvParams(3, op)
        p.conv_algo_desp = H.conv_desp(op, C, C)
        p.input, p.weight, p.output = inp, w, out
        back = "_bwd" if op == ConvOpType.BackwardInput else ""
        p.indices, p.mask, p.mask_argsort = (getattr(here, name + back) for name in names[:3])
        p.stream = stream.cuda_stream
        ConvMainUnitTest.implicit_gemm2(p)

    def passes(order, wait):
        made = []
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for i in order:
                y, din = torch.empty_like(x), torch.empty_like(x)
                for name in names:
                    getattr(here, name).copy_(getattr(scenes[i], name))
                x.copy_(rows[i])
                wait(stream)
                call(ConvOpType.Forward, x, y, stream)
                wait(stream)
                call(ConvOpType.BackwardInput, din, y, stream)
                wait(stream)
                made.append((y, din))
            stream.synchronize()
        H.check_status()
        return made

    want = passes(range(3), lambda s: s.synchronize())
    order = [0, 1, 2, 1, 0, 2, 0, 1]
    for i, got in zip(order, passes(order, lambda s: None)):
        assert torch.equal(got[0], want[i][0]) and torch.equal(got[1], want[i][1]), i


@pytest.mark.parametrize("max_ctas", [0, 4])
def test_tile_masks_of_launches_in_a_row_come_in_their_order(cuda_lib, max_ctas):
    """Two prepared forward calls over the fixed tables of two scenes, which report into one buffer.  The second is one
    that clusters share and that reads its tables while the first (such a call, too, or one whose four CTAs store their
    masks tile after tile) still runs: its masks are the ones that stay."""
    import torch
    from cumm_b200 import _lib
    from cumm_b200.layer import make_desp
    from cumm_b200.tensorview.gemm import ConvOpType, ConvParams, prepare_conv
    n, C, grid = 2000, 64, (8, 24, 24)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        masks = torch.zeros((n + 127) // 128, dtype=torch.int32, device="cuda")
        x, w = torch.zeros((n, C), dtype=torch.float16, device="cuda"), torch.zeros((C, 27, C), dtype=torch.float16, device="cuda")
        calls, wants = [], []
        for i, ctas in enumerate((max_ctas, 0)):
            tb = W.build_tables(W.sample_coords(n, 760 + i, grid), grid=grid)
            p = ConvParams(3, ConvOpType.Forward)
            p.conv_algo_desp = make_desp(ConvOpType.Forward, False, C, C)
            p.input, p.weight, p.output, p.mask_output = x, w, torch.zeros_like(x), masks
            p.indices, p.mask, p.mask_argsort = H.dev(tb.indices, torch), H.mask_to_torch(tb.mask, torch), H.dev(tb.mask_argsort, torch)
            p.max_ctas, p.stream = ctas, stream.cuda_stream
            p.mask_filter = 0xffffffff if i else 0x155
            calls.append(prepare_conv(p, static_tables=True))
            tile_masks = np.bitwise_or.reduceat(tb.mask & np.uint32(p.mask_filter), np.arange(0, n, 128))
            wants.append(H.mask_to_torch(tile_masks, torch))
        first, second = calls
        for c in calls + calls:
            c.launch()
        assert _lib.last_launch_info()["cluster"] == 4 and not torch.equal(*wants)
        for rounds in range(100):
            for c in (first, second, first, second) if rounds % 2 else (second, first, first, second):
                c.launch()
            assert torch.equal(masks, wants[1]), rounds
        first.launch()
        assert torch.equal(masks, wants[0])
    H.check_status()


def test_launches_behind_a_kernel_that_takes_longer_than_a_wait_may(cuda_lib):
    """A forward pass, over fixed tables and over tables that may be new, and a weight gradient with a plan of its own, each
    launched directly behind a forward pass that one CTA works at for 1.5 to 3 s.  They start beside it, and most of
    their warps wait for those that wait for its end: no wait has run out, results are those of launches on their own."""
    import torch
    from cumm_b200.conv.main import ConvMainUnitTest
    from cumm_b200.layer import DeviceTables, SparseConvLayer, make_desp
    from cumm_b200.tensorview.gemm import ConvOpType, ConvParams, prepare_conv
    half = lambda *s: torch.randn(s, device="cuda").half()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        C, K, kv = 1024, 2048, 27
        w = half(K, kv, C)

        def long_call(rows):
            p = ConvParams(3, ConvOpType.Forward)
            p.conv_algo_desp = make_desp(ConvOpType.Forward, False, C, K)
            p.input, p.weight, p.output = half(rows, C), w, torch.empty((rows, K), dtype=torch.float16, device="cuda")
            p.indices = torch.randint(0, rows, (kv, rows), dtype=torch.int32, device="cuda")
            p.mask = torch.full((rows,), (1 << kv) - 1, dtype=torch.int32, device="cuda")
            p.mask_argsort = torch.arange(rows, dtype=torch.int32, device="cuda")
            p.max_ctas, p.stream = 1, stream.cuda_stream
            return prepare_conv(p, static_tables=True)

        def seconds(call):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            call.launch()
            end.record()
            stream.synchronize()
            return begin.elapsed_time(end) / 1000

        few = 128 * 16
        trial = long_call(few)
        seconds(trial)
        long = long_call(int(few * 2 / seconds(trial)) // 128 * 128)
        tb = W.build_tables(W.sample_coords(9000, 770, (8, 48, 48)), grid=(8, 48, 48))
        n, c = tb.n_out, 64
        t = DeviceTables.from_host(tb, "cuda")
        x, dout, out, din = half(n, c), half(n, c), half(n, c), half(n, c)
        dw = half(c, 27, c)
        layer = SparseConvLayer(t, half(c, 27, c), x, out, dout, din, dw, stream=stream.cuda_stream)
        for call, result in ((layer.fwd.launch, out), (lambda: ConvMainUnitTest.implicit_gemm2(layer.fwd_params), out),
                             (layer.wgrad.launch, dw)):
            for _ in range(2):
                call()
            stream.synchronize()
            want = result.clone()
            result.zero_()
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            long.launch()
            call()
            end.record()
            stream.synchronize()
            assert 1.2 < begin.elapsed_time(end) / 1000 < 5
            H.check_status()
            assert torch.equal(result, want)


def test_a_prepared_call_is_ready_on_its_own_stream(cuda_lib):
    """Prepared while torch's own stream is busy and launched on the call's stream at once: the ticket counters are zero
    there, and neither they nor the scratch lie where memory of torch's stream was given back."""
    import torch
    from cumm_b200.layer import DeviceTables, SparseConvLayer
    t = DeviceTables.from_host(W.build_tables(W.sample_coords(20000, 780, (41, 100, 100)), grid=(41, 100, 100)), "cuda")
    half = lambda *s: (torch.randn(s, device="cuda") / 8).half()
    x, dout, w = half(t.n_in, 64), half(t.n_out, 64), half(64, 27, 64)
    big = half(8192, 8192)

    def launched(stream, busy):
        outs = torch.zeros_like(dout), torch.zeros_like(x), torch.zeros_like(w)
        ones = [torch.ones(n, dtype=torch.int32, device="cuda") for n in [8] * 6 + [1 << 20] * 6]
        torch.cuda.synchronize()
        for _ in range(busy):
            big @ big
        del ones  # free again, for torch's own stream
        layer = SparseConvLayer(t, w, x, outs[0], dout, outs[1], outs[2], stream=stream.cuda_stream)
        for call in (layer.fwd, layer.dgrad, layer.wgrad):
            call.launch()
            call.launch()
        stream.synchronize()
        assert not busy or not torch.cuda.current_stream().query()
        torch.cuda.synchronize()
        H.check_status()
        return outs

    want = launched(torch.cuda.current_stream(), 0)
    for rounds in range(3):
        for a, b in zip(launched(torch.cuda.Stream(), 30), want):
            assert torch.equal(a, b), rounds
