"""Quantiser and SwiGLU producer through the C ABI vs the CPU oracle (bit-exact)."""
import ctypes as C
import threading
import time

import numpy as np
import pytest
import torch

import oracle
from helpers import SEED, bits
from hygemm_vllm import fp4_quant, native, producer

pytestmark = pytest.mark.gpu

ROWS = [1, 3, 8, 17, 31, 32, 33, 64, 127, 128, 129, 255, 256, 257]


def _random(rows, k, dtype, scale, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(rows, k, generator=g) * scale
    x[:, ::53] *= 20
    if rows > 2:
        x[1, :64] = 0                      # all-zero K32 blocks
        x[2, 5] = -0.0
    return x.to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("fp4", [False, True])
def test_pack_is_bit_exact_incl_padding(dtype, fp4):
    """Matrix of optimization/check_pack.py:17-35 of the reference (rows x K x scales), codes AND
    the whole scale buffer, with the buffer pre-filled with 0xff so stale padding would show."""
    for rows in ROWS:
        for k, scale in [(128, 0.125), (896, 2.0), (3584, 1.0)]:
            x = _random(rows, k, dtype, scale, rows * 7 + k)
            xd = x.cuda()
            q, sf = native.pack(xd, fp4)
            sf.fill_(255)
            q2, sf2 = native.pack(xd, fp4)          # second call must rewrite every byte
            want_q, want_sf = oracle.pack(x, fp4=fp4, bf16=dtype == torch.bfloat16)
            assert np.array_equal(q2.cpu().numpy(), want_q), (rows, k)
            assert np.array_equal(sf2.cpu().numpy(), want_sf), (rows, k)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_pack_every_finite_16bit_value(dtype):
    """Every finite bit pattern as an input and as a group maximum
    (performance/check.py:39-44, performance/check_pack_maxima.py:9-22 of the reference)."""
    allbits = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(dtype)
    finite = allbits[torch.isfinite(allbits.float())]
    pad = (-finite.numel()) % 128
    x = torch.cat([finite, finite[:pad]]).reshape(-1, 128)
    for fp4 in (False, True):
        q, sf = native.pack(x.cuda(), fp4)
        want_q, want_sf = oracle.pack(x, fp4=fp4, bf16=dtype == torch.bfloat16)
        assert np.array_equal(q.cpu().numpy(), want_q)
        assert np.array_equal(sf.cpu().numpy(), want_sf)
    # each value as the maximum of an otherwise tiny group (scale-boundary ties)
    vals = finite[finite.float().abs() > 0][::3]
    rows = vals.numel()
    x = torch.zeros(rows, 128, dtype=dtype)
    x[:, 0] = vals
    x[:, 1] = (vals.float() * 0.37).to(dtype)
    x[:, 33] = vals
    x[:, 40] = -(vals.float() * 0.5).to(dtype)
    q, sf = native.pack(x.cuda(), False)
    want_q, want_sf = oracle.pack(x, fp4=False, bf16=dtype == torch.bfloat16)
    assert np.array_equal(q.cpu().numpy(), want_q)
    assert np.array_equal(sf.cpu().numpy(), want_sf)


@pytest.mark.parametrize("fp4", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_16bit_value_as_the_maximum_of_a_group(dtype, fp4):
    """Codes and scale bytes of both formats, so the values just below and above each 1.5 x 2^n and 1.75 x 2^n are among them; the exponent
    search without offsets starts from the same exponents."""
    everything = torch.arange(1, 1 << 15, dtype=torch.int32).to(torch.int16).view(dtype)
    values = everything[torch.isfinite(everything.float())]
    values = torch.cat([values, values.new_zeros(-values.numel() % 4)])
    groups = torch.zeros(values.numel(), 32, dtype=dtype)
    for column, factor in ((0, 1.0), (7, -0.5), (13, 0.37), (31, -0.08)):
        groups[:, column] = (values.float() * factor).to(dtype)
    x = groups.view(-1, 128)
    q, sf = native.pack(x.cuda(), fp4)
    want_q, want_sf = oracle.pack(x, fp4=fp4, bf16=dtype == torch.bfloat16)
    assert np.array_equal(sf.cpu().numpy(), want_sf) and np.array_equal(q.cpu().numpy(), want_q)
    if fp4:
        codes, scales, _ = fp4_quant.quantize(x.cuda(), offsets=())
        assert np.array_equal(codes.cpu().numpy(), want_q)
        assert np.array_equal(scales.cpu().numpy(), want_sf[oracle.scale_indices(*x.shape)])


def test_fp4_tie_table():
    """allocation/check_components.py:14 of the reference: exact ties and signed zeros."""
    ties = [0., -0., .25, .75, 1.25, 1.75, 2.5, 3.5, 5., 6., -.25, -.75, -1.25, -1.75, -2.5, -3.5, -5., -6.]
    x = torch.zeros(1, 128, dtype=torch.float16)
    x[0, :len(ties)] = torch.tensor(ties, dtype=torch.float16)
    x[0, 31] = 6.0
    q, sf = native.pack(x.cuda(), True)
    want_q, want_sf = oracle.pack(x, fp4=True, bf16=False)
    assert np.array_equal(q.cpu().numpy(), want_q) and np.array_equal(sf.cpu().numpy(), want_sf)


def test_pack_rejects_bad_arguments():
    x = torch.zeros(4, 100, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ValueError):
        native.pack(x)
    lib = native.library()
    assert lib.hg_pack(None, None, None, 1, 128, 0, None) == -1
    assert b"Invalid MX pack arguments" in lib.hg_last_error()
    assert lib.hg_silu_pack(None, None, None, None, 1, 128, None, 0) == 1     # cudaErrorInvalidValue


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_silu_pack_matches_oracle_and_two_step_path(dtype):
    """performance/check_producer.py:17-28 of the reference: codes, scales and the 16-bit product of the
    fused kernel equal SiluAndMul followed by pack.  expf differs by <= 1 ulp between CPU and GPU libraries,
    so the CPU comparison allows rare 16-bit neighbours; the quantisation of the device's own product
    must be bit-exact."""
    bf16 = dtype == torch.bfloat16
    for rows, k, scale in [(1, 128, 1.0), (3, 896, 4.0), (33, 4864, 0.1), (128, 18944, 2.0), (129, 896, 16.0)]:
        g = torch.Generator().manual_seed(rows + k)
        x = (torch.randn(rows, 2 * k, generator=g) * scale).to(dtype)
        q, sf, dbg = producer.silu_pack(x.cuda(), 0, debug=True)
        oq, osf, odbg = oracle.silu_pack(x, bf16=bf16, debug=True)
        got = bits(dbg)
        differ = got != odbg
        assert differ.mean() < 1e-3, (rows, k, differ.mean())
        # neighbours only
        assert np.all(np.abs(got[differ].astype(np.int32) - odbg[differ].astype(np.int32)) <= 1)
        q2, sf2 = oracle.pack(dbg.cpu(), fp4=False, bf16=bf16)
        assert np.array_equal(q.cpu().numpy(), q2) and np.array_equal(sf.cpu().numpy(), sf2), (rows, k)
        # two-step device path: torch SiLU*up (same expf library) then hg_pack
        xd = x.cuda()
        act = torch.nn.functional.silu(xd[:, :k].float()).to(dtype)
        prod = (act.float() * (xd[:, k:].float() + 0.0)).to(dtype)
        q3, sf3 = native.pack(prod.contiguous())
        same = (bits(prod) == got).mean()
        assert same > 0.999, (rows, k, same)
        if same == 1.0:
            assert torch.equal(q3, q) and torch.equal(sf3, sf)


def test_silu_pack_vs_vllm_op():
    """Bitwise parity with the installed vLLM SiluAndMul op followed by pack, when that op is available."""
    try:
        import vllm._custom_ops  # noqa: F401
        op = torch.ops._C.silu_and_mul
    except Exception:
        pytest.skip("vLLM custom ops not loadable")
    for dtype in (torch.bfloat16, torch.float16):
        for rows, k in [(1, 128), (33, 896), (128, 18944)]:
            g = torch.Generator().manual_seed(rows * 3 + k)
            x = (torch.randn(rows, 2 * k, generator=g) * 2).to(dtype).cuda()
            out = torch.empty(rows, k, dtype=dtype, device="cuda")
            op(out, x)
            q_ref, sf_ref = native.pack(out)
            q, sf, dbg = producer.silu_pack(x, 0, debug=True)
            assert torch.equal(dbg.view(torch.int16), out.view(torch.int16)), (dtype, rows, k)
            assert torch.equal(q, q_ref) and torch.equal(sf, sf_ref)


def _specials(x, seed):
    """The same matrix with infinities, NaNs, whole groups of them, zeros and the smallest values, about one group in fifty."""
    g = torch.Generator().manual_seed(seed)
    x = x.clone()
    groups = x.view(-1, 32)
    picked = torch.randperm(groups.shape[0], generator=g)[: max(8, groups.shape[0] // 50)].split(max(1, groups.shape[0] // 400))
    for rows, value in zip(picked, (float("inf"), float("-inf"), float("nan"), 0.0, -0.0, torch.finfo(x.dtype).tiny, torch.finfo(x.dtype).smallest_normal / 4,
                                    torch.finfo(x.dtype).max)):
        half = rows[: rows.numel() // 2]
        groups[half] = value
        groups[rows, torch.randint(0, 32, (rows.numel(),), generator=g)] = value
    return x


# 4 M elements and more (SwiGLU: 8 M products) take the kernels with four rows a warp; K that is no multiple of their 512 columns, and
# rows that end inside a 128-row scale block, in each of its quarters.
MANY_ROWS = [(777, 18944), (4128 - 31, 2176), (65600, 128), (33000, 256), (4096, 2048)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,k", MANY_ROWS)
def test_many_rows_equal_few_rows_and_the_oracle(rows, k, dtype):
    """`pack` and the SwiGLU producer on a large matrix against the oracle, and against the kernels for few rows on its
    128-row blocks (infinities and NaNs too, which the oracle does not define)."""
    assert rows * k >= 8 << 20
    bf16 = dtype == torch.bfloat16
    x = _random(rows, k, dtype, 1.0, rows + k)
    for fp4 in (False, True):
        q, sf = native.pack(x.cuda(), fp4)
        want_q, want_sf = oracle.pack(x, fp4=fp4, bf16=bf16)
        assert np.array_equal(q.cpu().numpy(), want_q) and np.array_equal(sf.cpu().numpy(), want_sf), fp4
        special = _specials(x, rows).cuda()
        chunks = [native.pack(c.contiguous(), fp4) for c in special.split(128)]
        q, sf = native.pack(special, fp4)
        assert torch.equal(q, torch.cat([c[0] for c in chunks])) and torch.equal(sf, torch.cat([c[1] for c in chunks])), fp4
        if rows * k < 16 << 20:
            shifted = torch.empty(rows * k + 8, dtype=dtype, device="cuda")[8:].view(rows, k).copy_(special)   # 16 bytes off: no 32-byte loads
            other = native.pack(shifted, fp4)
            assert torch.equal(q, other[0]) and torch.equal(sf, other[1]), fp4
    gate = _random(rows, k, dtype, 2.0, rows + k + 1)
    pair = torch.cat([gate, x], 1).cuda()
    q, sf, product = producer.silu_pack(pair, 0, debug=True)
    want_q, want_sf = oracle.pack(product.cpu(), bf16=bf16)
    assert np.array_equal(q.cpu().numpy(), want_q) and np.array_equal(sf.cpu().numpy(), want_sf)
    fast = producer.silu_pack(pair, 0)
    assert torch.equal(fast[0], q) and torch.equal(fast[1], sf)
    for math in (0, 1, 2):
        pair = torch.cat([_specials(gate, rows + 1), _specials(x, rows + 2)], 1).cuda()
        chunks = [producer.silu_pack(c.contiguous(), math) for c in pair.split(128)]
        q, sf = producer.silu_pack(pair, math)
        assert torch.equal(q, torch.cat([c[0] for c in chunks])) and torch.equal(sf, torch.cat([c[1] for c in chunks])), math


def test_split_verdict_belongs_to_the_maps_that_are_packed():
    """Maps made in one order and packed in another, and maps that are never packed: every packing reports on its own maps."""
    lib, stream = native.library(), torch.cuda.current_stream().cuda_stream
    rows, k = 300, 256
    weight = torch.randn(rows, k, generator=torch.Generator().manual_seed(SEED)).bfloat16().cuda()
    lists = {"repeated": [7, 7, 9, 250], "out of range": [3, 300, 5, -1], "good": [299, 0, 31, 32], "none": [], "all": list(range(rows))[::-1],
             "last one repeated": [5, 6, 299, 299], "all but one": [0, *range(rows - 1)]}
    distinct = {"repeated": (3, 0), "out of range": (2, 1), "good": (4, 0), "none": (0, 0), "all": (rows, 0), "last one repeated": (3, 0),
                "all but one": (rows - 1, 0)}

    def maps(name):
        ids = torch.tensor(lists[name], dtype=torch.int64).cuda()
        hi = torch.full((len(lists[name]),), 1 << 30, dtype=torch.int32, device="cuda")
        lo = torch.full((rows - len(lists[name]),), 1 << 30, dtype=torch.int32, device="cuda")
        native.check(lib.hg_split_rows(ids.data_ptr(), ids.numel(), rows, lo.data_ptr(), hi.data_ptr(), stream))
        torch.cuda.synchronize()
        return lo, hi

    made = {name: maps(name) for name in lists}
    for name in reversed(lists):
        lo, hi = made[name]
        n = hi.numel()
        w4, w8 = (torch.empty(s, dtype=torch.uint8, device="cuda") for s in ((rows - n, k // 2), (n, k)))
        sf4, sf8 = (torch.empty(native.scale_size(r, k), dtype=torch.uint8, device="cuda") for r in (rows - n, n))
        verdict = (C.c_int * 2)()
        native.check(lib.hg_split_pack(weight.data_ptr(), n, rows, k, lo.data_ptr(), hi.data_ptr(), w4.data_ptr(), sf4.data_ptr(), w8.data_ptr(),
                                       sf8.data_ptr(), verdict, 1, stream))
        assert tuple(verdict) == distinct[name], name
        if verdict[0] == n and not verdict[1]:
            assert hi.tolist() == sorted(lists[name]) and lo.tolist() == sorted(set(range(rows)) - set(lists[name]))
            for part, codes, sf, fp4 in ((lo, w4, sf4, True), (hi, w8, sf8, False)):
                want, want_sf = native.pack(weight[part.long()].contiguous(), fp4)
                assert torch.equal(codes, want) and torch.equal(sf, want_sf)


def test_calls_with_a_host_result_beside_a_capture_and_from_many_threads():
    """Packing and offline search end with numbers for the host.  A thread that made such calls and ends, or makes its first ones, does
    not disturb a capture on another thread; calls of many threads at once each get their own numbers."""
    w = (torch.randn(256, 256, generator=torch.Generator().manual_seed(SEED)) * 0.03).bfloat16().cuda()
    ids = torch.arange(0, 256, 5).cuda()
    _, _, want = fp4_quant.quantize(w)
    may_end, made, failures = threading.Event(), threading.Barrier(9), []

    def worker(index):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                scale = 2.0 ** index                         # an exact factor of the weights: its square in the errors
                mine = w * scale
                torch.cuda.current_stream().synchronize()
                for _ in range(20):
                    _, _, stats = fp4_quant.quantize(mine)
                    assert stats["shift_groups"] == want["shift_groups"]
                    for name in ("weight_error_before", "weight_error_after"):
                        # the same terms, in another order: 8192 of them in fp64
                        assert abs(stats[name] / (scale * scale * want[name]) - 1) < 1e-11
                layer = native.DualLinear(mine, ids)
                assert torch.equal(layer.hi.long(), ids)
                layer.close()
        except Exception as e:   # noqa: BLE001
            failures.append(e)
        made.wait()
        may_end.wait()

    threads = [threading.Thread(target=worker, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    made.wait()
    assert not failures, failures
    x = torch.ones(16, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = x + 1
        may_end.set()
        for t in threads:
            t.join()
        time.sleep(0.5)                                      # the threads themselves end a little after their joins
        y = y + 1
    graph.replay()
    assert torch.equal(y, x + 2)
