"""The cluster GEMM where its plan changes: token counts on both sides of every tile width and of the single / paired CTA
switch, K with odd and single K128 blocks (also cut over a cluster), row counts around a tile.

Operands are exactly representable and their sums stay below 2^24 quanta, so every order of summation gives the same fp32
value: results must be equal bit for bit (tolerance 0).
"""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
from helpers import expected_work, run_gemm, swiglu_unit_probe
from hygemm_vllm import native, producer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 16, 17, 32, 33, 64, 65, 96, 127, 129, 255, 257, 290])
def test_exact_at_the_edges_of_the_plan(tokens):
    for outputs, k, high in [(129, 128, 1), (640, 896, 128), (385, 2432, 129)]:
        case = oracle.exact_case(outputs, tokens, k, high, "random")
        got, guards, status = run_gemm(case, torch.bfloat16, 0)
        assert status[0] == 0 and guards, (outputs, k, high, status)
        assert (status[1], status[2]) == expected_work(case, 0), (outputs, k, high, status)
        assert np.array_equal(got, case["expected"]), (outputs, k, high, int((got != case["expected"]).sum()))


@pytest.mark.parametrize("tokens,k,forced", [(2048, 384, False), (1990, 896, False), (1825, 128, False), (777, 384, True), (290, 256, True)])
def test_exact_with_several_wide_tiles_per_cluster(tokens, k, forced, monkeypatch):
    """256-token tiles: their two accumulators share 32 TMEM columns, which are handed from one to the other early.  That happens from a
    cluster's second unit on, so every cluster has at least two here, with tails of every kind of width."""
    if forced:
        monkeypatch.setenv("HYGEMM_CL_N", "256")
    outputs, high = (8269, 800) if tokens > 512 else (18944, 1900)
    case = oracle.exact_case(outputs, tokens, k, high, "random")
    header = (C.c_int * 12)()
    native.check(native.library().hg_plan(outputs - high, high, tokens, k, torch.cuda.get_device_properties(0).multi_processor_count, 0, header, None, 0))
    assert header[2] == 256 and header[9] >= 1.9 * header[1], list(header)   # units per CTA
    got, guards, status = run_gemm(case, torch.bfloat16, 0)
    assert status[0] == 0 and guards and (status[1], status[2]) == expected_work(case, 0)
    assert np.array_equal(got, case["expected"]), int((got != case["expected"]).sum())


@pytest.mark.parametrize("tokens,width", [(129, 160), (160, 160), (193, 224), (300, 192), (310, 256), (450, 192), (577, 224), (641, 192), (777, 224), (1000, 192)])
def test_exact_in_tiles_that_fit_a_ragged_prompt(tokens, width, monkeypatch):
    """One tile of up to 256 tokens, steps of 192 whose every second tile starts in the middle of a scale atom, a last tile joined to the one
    before it (wider than the others, over three scale atoms): one and several units to a cluster, whole and cut along K."""
    monkeypatch.setenv("HYGEMM_CL_N", str(width))
    for (outputs, k, high), split in [((8269, 384, 800), 1), ((640, 896, 128), 1), ((640, 896, 128), 2), ((18944, 128, 1000), 1)]:
        if split > 1 and width > 224:
            continue   # 256 tokens are never cut along K
        monkeypatch.setenv("HYGEMM_CL_SPLIT", str(split))
        case = oracle.exact_case(outputs, tokens, k, high, "random")
        got, guards, status = run_gemm(case, torch.bfloat16, 0)
        assert status[0] == 0 and guards and (status[1], status[2]) == expected_work(case, 0), (outputs, k, high, split, status)
        assert np.array_equal(got, case["expected"]), (outputs, k, high, split, int((got != case["expected"]).sum()))


@pytest.mark.parametrize("tokens", [801, 820, 832])
@pytest.mark.parametrize("outputs,k,high", [(8269, 384, 800), (18944, 128, 1000), (18944, 1152, 2000)])
def test_exact_with_a_last_tile_of_256_tokens_behind_tiles_of_192(outputs, k, high, tokens, monkeypatch):
    """Steps of 192 with what is left joined to the last one: two accumulators that share columns serve tiles of unlike width, and 256
    columns start in the middle of a scale atom and read three.  Every cluster has several units; steps of 256 would need two atoms."""
    monkeypatch.setenv("HYGEMM_CL_N", "256")
    case = oracle.exact_case(outputs, tokens, k, high, "random")
    header = (C.c_int * 12)()
    native.check(native.library().hg_plan(outputs - high, high, tokens, k, torch.cuda.get_device_properties(0).multi_processor_count, 0, header, None, 0))
    assert list(header[2:6]) == [256, 4, 3, 210208] and header[9] >= 1.9 * header[1], list(header)
    got, guards, status = run_gemm(case, torch.bfloat16, 0)
    assert status[0] == 0 and guards and (status[1], status[2]) == expected_work(case, 0), status
    assert np.array_equal(got, case["expected"]), int((got != case["expected"]).sum())


@pytest.mark.parametrize("pair", [1, 2])
@pytest.mark.parametrize("split", [1, 2, 4])
@pytest.mark.parametrize("tokens", [65, 80, 97, 128])
def test_exact_in_two_tiles_of_64_tokens(tokens, split, pair, monkeypatch):
    """65 to 128 tokens as two tiles, the second of which starts in the middle of its scale atom: single and paired CTAs, whole and cut
    along K, one unit per cluster and (the last shape, uncut) several."""
    for name, value in (("N", 64), ("PAIR", pair), ("SPLIT", split)):
        monkeypatch.setenv("HYGEMM_CL_" + name, str(value))
    for outputs, k, high in [(129, 1152, 1), (640, 896, 128)] + [(18944, 384, 1000)] * (split == 1):
        case = oracle.exact_case(outputs, tokens, k, high, "random")
        header = (C.c_int * 12)()
        native.check(native.library().hg_plan(outputs - high, high, tokens, k, torch.cuda.get_device_properties(0).multi_processor_count, 0, header, None, 0))
        assert (header[2], header[3]) == (64, 2), list(header)
        got, guards, status = run_gemm(case, torch.bfloat16, 0)
        assert status[0] == 0 and guards and (status[1], status[2]) == expected_work(case, 0), (outputs, k, high, status)
        assert np.array_equal(got, case["expected"]), (outputs, k, high, int((got != case["expected"]).sum()))


@pytest.mark.parametrize("tokens,pair,split", [(t, p, s) for t, p in [(17, 1), (33, 1), (36, 2), (50, 1), (64, 2), (100, 2), (128, 2)]
                                               for s in (2, 4, 8) if p * s <= 8])
def test_exact_cut_along_k_at_every_way_of_the_exchange(tokens, pair, split, monkeypatch):
    """Partial sums of one token tile on all their ways through a cluster: asynchronous stores up to 32 tokens, above that through the ring,
    with slices of one K128 block and of unequal length, partitions that end inside a tile and tiles of 128, 64 and 32 rows."""
    width = -(-tokens // (16 * pair)) * 16 * pair
    for name, value in (("N", width), ("PAIR", pair), ("SPLIT", split)):
        monkeypatch.setenv("HYGEMM_CL_" + name, str(value))
    for (outputs, k, high), cut in [((129, 128 * (2 * split - 1), 1), 0), ((640, 2432, 128), 1), ((257, 3200, 1), 2)]:
        monkeypatch.setenv("HYGEMM_CL_CUT", str(cut))
        case = oracle.exact_case(outputs, tokens, k, high, "random")
        for _ in range(3):
            got, guards, status = run_gemm(case, torch.bfloat16, 0)
            assert status[0] == 0 and guards and (status[1], status[2]) == expected_work(case, 0), (outputs, k, high, status)
            assert np.array_equal(got, case["expected"]), (outputs, k, high, int((got != case["expected"]).sum()))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_swiglu_layer_call_equals_producer_then_gemm(dtype):
    """One foreign call for SwiGLU and down_proj: the same bytes as the producer followed by the GEMM on its codes."""
    g = torch.Generator().manual_seed(3)
    for outputs, k, high in [(257, 128, 26), (300, 896, 0), (640, 2432, 128), (384, 256, 384)]:
        layer = native.DualLinear((torch.randn(outputs, k, generator=g) * 0.04).to(dtype).cuda(), torch.randperm(outputs, generator=g)[:high].cuda())
        for tokens in (1, 8, 17, 130):
            x = torch.randn(tokens, 2 * k, generator=g) * 2
            x[0, :64] = 0
            x = x.to(dtype).cuda()
            got = layer.silu_linear(x, 0)
            want = layer.run_packed(*producer.silu_pack(x, 0))
            assert torch.equal(got.view(torch.int16), want.view(torch.int16)), (outputs, k, high, tokens)
        assert layer.status()[0] == 0
        layer.close()


@pytest.mark.parametrize("tokens", [1, 16, 17, 130])
def test_layer_call_by_every_route(tokens):
    """Prepared calls, the first call, the other input dtype, tensor subclasses, replaced weights and a changed
    schedule id: always the bytes of the quantiser followed by the GEMM on its codes, and one count per call."""
    g = torch.Generator().manual_seed(tokens)
    outputs, k, high = 300, 384, 40
    layer = native.DualLinear((torch.randn(outputs, k, generator=g) * 0.04).half().cuda(), torch.arange(high).cuda())
    wide = torch.randn(tokens, 2 * k, generator=g).half().cuda()
    x = wide[:, :k].contiguous()

    def check(x):
        before = layer.calls.get(tokens, 0)
        got = layer(x)
        assert layer.calls[tokens] == before + 1 and got.dtype == torch.float16 and type(got) is torch.Tensor
        assert torch.equal(got.view(torch.int16), layer.run_packed(*native.pack(x.contiguous())).view(torch.int16))
        return got

    check(x), check(x)
    check(x.bfloat16())
    check(torch.nn.Parameter(x, requires_grad=False))
    layer.w4, layer.sf4 = layer.w4.flip(0).contiguous(), layer.sf4.clone()
    torch.cuda.synchronize()
    check(x), check(x)
    layer.low_id = layer.high_id = 1
    check(x), check(x)
    for bad in (wide, x.cpu(), x[0], wide[:, ::2]):
        with pytest.raises(ValueError):
            layer(bad)
    layer.close()


def test_layer_calls_without_the_host_extension(monkeypatch):
    """A library whose host extension was not built: the layer says so once it is made, and its calls give the same bytes."""
    g = torch.Generator().manual_seed(5)
    w, ids = (torch.randn(300, 256, generator=g) * 0.04).bfloat16().cuda(), torch.arange(40).cuda()
    x, pair = torch.randn(5, 256, generator=g).bfloat16().cuda(), torch.randn(5, 512, generator=g).bfloat16().cuda()
    layer = native.DualLinear(w, ids)
    want = layer(x), layer.silu_linear(pair, 0)
    monkeypatch.setattr(native, "_host", None)
    with pytest.warns(RuntimeWarning, match="host extension not found"):
        plain = native.DualLinear(w, ids)
    assert torch.equal(plain(x), want[0]) and torch.equal(plain.silu_linear(pair, 0), want[1])
    layer.close()
    plain.close()


@pytest.mark.parametrize("how", ["attribute", "storage"])
@pytest.mark.parametrize("name", ["w4", "sf4", "lo", "w8", "sf8", "hi"])
def test_layer_call_after_an_operand_was_replaced(name, how):
    """Each operand tensor of a layer exchanged, as an attribute and as the storage behind it, after calls that prepared the layer:
    the bytes of a layer that had the new operand from the start, by the one-call route and by `run_packed`."""
    g = torch.Generator().manual_seed(11)
    outputs, k, high = 300, 384, 40

    def fresh(seed):
        g.manual_seed(seed)
        return native.DualLinear((torch.randn(outputs, k, generator=g) * 0.04).bfloat16().cuda(), torch.randperm(outputs, generator=g)[:high].cuda())

    layer, other, wanted = fresh(1), fresh(2), fresh(1)
    new = getattr(layer, name).flip(0).contiguous() if name in ("lo", "hi") else getattr(other, name)
    setattr(wanted, name, new)
    for tokens in (3, 40):
        x = torch.randn(tokens, k, generator=g).bfloat16().cuda()
        y, want = layer(x), wanted(x)
        assert torch.equal(y, layer.run_packed(*native.pack(x))) and not torch.equal(y, want)
        old = getattr(layer, name).clone()
        if how == "attribute":
            setattr(layer, name, new.clone())
        else:
            getattr(layer, name).data = new.clone()
        torch.cuda.synchronize()
        assert torch.equal(layer(x), want) and torch.equal(layer.run_packed(*native.pack(x)), want)
        setattr(layer, name, old)
        torch.cuda.synchronize()
        assert torch.equal(layer(x), y)
    for each in (layer, other, wanted):
        each.close()


@pytest.mark.parametrize("schedule", [0, 1])
def test_status_of_a_handle_made_on_a_busy_stream(schedule):
    """A handle made on one stream and run on another: its status words are clear before it is handed out, so the launch's counts
    are not cleared behind its back."""
    lib = native.library()
    g = torch.Generator().manual_seed(8)
    layer = native.DualLinear((torch.randn(300, 256, generator=g) * 0.04).bfloat16().cuda(), torch.arange(40).cuda())
    q, sf = native.pack(torch.randn(5, 256, generator=g).bfloat16().cuda())
    y = torch.empty(5, 300, dtype=torch.bfloat16, device="cuda")
    low, high = layer.problems(q, sf, y)
    layer.low_id = layer.high_id = schedule
    layer.run_packed(q, sf)   # the kernel is loaded
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(200_000_000)   # about a tenth of a second
    handle = C.c_void_p()
    native.check(lib.hg_create_dtype(schedule, schedule, C.byref(low), C.byref(high), busy.cuda_stream, 1, C.byref(handle)))
    native.check(lib.hg_run(handle, C.byref(low), C.byref(high), other.cuda_stream, 0))
    torch.cuda.synchronize()
    status = (C.c_int * 3)()
    native.check(lib.hg_status(handle, other.cuda_stream, status))
    lib.hg_destroy(handle)
    layer.close()
    assert status[0] == 0 and status[1] > 0 and status[2] > 0, list(status)


def test_swiglu_layer_refuses_an_unknown_math():
    """What the producer refuses stays refused on a prepared layer: not taken for the layer on an input that is as wide as its K."""
    g = torch.Generator().manual_seed(6)
    layer = native.DualLinear((torch.randn(300, 256, generator=g) * 0.04).bfloat16().cuda(), torch.arange(40).cuda())
    x, pair = torch.randn(5, 256, generator=g).bfloat16().cuda(), torch.randn(5, 512, generator=g).bfloat16().cuda()
    layer(x), layer.silu_linear(pair, 0)
    calls = dict(layer.calls)
    for math in (-1, -7, 3):
        for given in (x, pair):
            with pytest.raises(RuntimeError, match="producer"):
                layer.silu_linear(given, math)
    assert layer.calls == calls
    layer.close()


@pytest.mark.parametrize("policy", [False, True, 0, 2, 3, 4, 5, 6, 7, -1])
def test_layer_calls_keep_the_launch_policy(policy):
    """`layer(x)` and `silu_linear` under every launch policy, set when the layer is built and changed after calls that prepared it:
    the bytes of `run_packed`, which the GEMV policies send to the SIMT kernel; unknown policies are refused by both."""
    g = torch.Generator().manual_seed(4)
    outputs, k, high = 300, 2432, 40
    w, ids = (torch.randn(outputs, k, generator=g) * 0.04).bfloat16().cuda(), torch.arange(high).cuda()
    built, changed = native.DualLinear(w, ids, concurrent=policy), native.DualLinear(w, ids)
    for tokens in (3, 40):
        x = torch.randn(tokens, k, generator=g).bfloat16().cuda()
        pair = torch.randn(tokens, 2 * k, generator=g).bfloat16().cuda()
        changed.concurrent = True
        changed(x), changed.silu_linear(pair, 0)
        changed.concurrent = policy
        for layer in (built, changed):
            if policy in (7, -1):
                for call in (lambda: layer(x), lambda: layer.silu_linear(pair, 0), lambda: layer.run_packed(*native.pack(x))):
                    with pytest.raises(RuntimeError, match="Unknown launch policy"):
                        call()
                continue
            layer.status()
            for call, packed in ((lambda: layer(x), native.pack(x)), (lambda: layer.silu_linear(pair, 0), producer.silu_pack(pair, 0))):
                y = call()
                assert (layer.status()[1] > 0) == (policy not in (4, 5, 6))   # K128 blocks that the tensor cores were given
                assert torch.equal(y, layer.run_packed(*packed))
                layer.status()
    built.close()
    changed.close()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_swiglu_of_every_gate_value(dtype):
    """Both SwiGLU producers (many rows, few rows) on all 65536 gates of the type, infinities and NaNs too, each with 128 values of
    up: the bytes of the producer that also returns its products, which keeps to the exact functions."""
    k = 2048
    g = torch.Generator(device="cuda").manual_seed(9)
    gate = torch.arange(65536, device="cuda").repeat(128)[torch.randperm(128 * 65536, device="cuda", generator=g)]
    up = torch.randint(0, 65536, (128 * 65536,), device="cuda", generator=g)
    gate, up = (t.to(torch.int16).view(dtype).view(-1, k) for t in (gate, up))
    up = torch.where(torch.arange(up.shape[0], device="cuda")[:, None] % 4 == 0, up, torch.randn(up.shape, device="cuda", generator=g).to(dtype))
    x = torch.cat([gate, up], 1).contiguous()
    for part in (x, *x.split(512)):
        q, sf = producer.silu_pack(part, 0)
        exact_q, exact_sf, _ = producer.silu_pack(part, 0, debug=True)
        assert torch.equal(q, exact_q) and torch.equal(sf, exact_sf)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_swiglu_of_every_gate_to_the_last_unit(dtype):
    """The producers' activations of all finite gates, wide and narrow window around rounding boundaries, are the exact functions' to the last
    of their 16 bits: a gate has a K32 group to itself and values of up with which one unit shows in its bytes (tolerance 0; the CPU test of
    `swiglu_unit_probe` plants the unit).  One row of 1024, few rows, many rows (from 8 Mi elements) and, wide and of 33 rows or more, in place."""
    gate = torch.arange(65536, device="cuda").to(torch.int16).view(dtype)
    gate = gate[torch.isfinite(gate)].sort().values
    gate = torch.cat([gate, gate[:-gate.numel() % 2304]])
    up, _ = swiglu_unit_probe(gate)
    pairs = torch.stack([gate[:, None].expand_as(up), up])
    for k, rows in ((1024, 1), (1024, 300), (1024, 8208), (9216, 57)):
        part = pairs.reshape(2, -1, k)
        part = torch.cat([part[0], part[1]], 1)
        part = part.repeat(-(-rows // part.shape[0]), 1)
        for x in part[:8].split(1) if rows == 1 else part.split(rows):
            q, sf = producer.silu_pack(x, 0)
            exact_q, exact_sf, _ = producer.silu_pack(x, 0, debug=True)
            assert torch.equal(q, exact_q) and torch.equal(sf, exact_sf), (k, rows)


@pytest.mark.parametrize("rows,k", [(32, 9216), (33, 9088), (33, 9216), (67, 9216), (68, 9216), (33, 18688), (33, 18816)])
def test_swiglu_where_doubtful_pairs_are_taken_in_place(rows, k):
    """Around the edges of the rule (33 rows, 9216 channels, 302 blocks of 2048 elements), both types: the exact functions' bytes."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    for dtype in (torch.float16, torch.bfloat16):
        x = (torch.randn(rows, 2 * k, device="cuda", generator=g) * 5).to(dtype)
        q, sf = producer.silu_pack(x, 0)
        exact_q, exact_sf, _ = producer.silu_pack(x, 0, debug=True)
        assert torch.equal(q, exact_q) and torch.equal(sf, exact_sf)


@pytest.mark.parametrize("tokens", [1, 2, 7, 8, 9, 16])
@pytest.mark.parametrize("outputs,k,high", [(19900, 384, 1900), (20000, 1408, 1), (640, 3712, 64), (300, 128, 30)])
def test_quantisation_in_the_gemm_over_several_units(outputs, k, high, tokens):
    """Several units to a CTA, K of fewer and of more steps than a quantiser has on the way and no multiple of them, eager and captured:
    the bytes of the quantiser followed by the GEMM (the same arithmetic: tolerance 0)."""
    g = torch.Generator(device="cuda").manual_seed(tokens)
    for dtype in (torch.bfloat16, torch.float16):
        w = torch.randn(outputs, k, device="cuda", generator=g, dtype=dtype) * 0.04
        layer = native.DualLinear(w, torch.randperm(outputs, device="cuda", generator=g)[:high])
        x = torch.randn(tokens, k, device="cuda", generator=g).to(dtype)
        x[:, ::97] *= 20
        want = layer.run_packed(*native.pack(x))
        y = torch.empty_like(want)
        low, hi = layer.problems(x, x, y)   # in the GEMM at every token count
        handle = layer.handles[next(iter(layer.handles))]
        stream = torch.cuda.current_stream().cuda_stream
        native.check(native.library().hg_run_x(handle, C.byref(low), C.byref(hi), x.data_ptr(), native.DTYPES[dtype], stream))
        assert torch.equal(y.view(torch.int16), want.view(torch.int16)) and torch.equal(layer(x).view(torch.int16), want.view(torch.int16))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = layer(x)
        x.mul_(2)
        graph.replay()
        assert torch.equal(captured.view(torch.int16), layer.run_packed(*native.pack(x)).view(torch.int16))
        assert layer.status()[0] == 0
        layer.close()
