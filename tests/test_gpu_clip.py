"""Offline MXFP4 exponent search (hg_clip_pack / fp4_quant.quantize) against the CPU oracle: bit-exact codes
and scale bytes, on the committed golden inputs and on larger seeded matrices of both dtypes."""
import numpy as np
import pytest
import torch

import oracle
from helpers import SEED, dev
from hygemm_vllm import fp4_quant, native, offline_weights

pytestmark = pytest.mark.gpu
GOLDEN = np.load(__import__("pathlib").Path(__file__).parent / "golden" / "clip_search.npz")


@pytest.mark.parametrize("tag", ["plain", "weighted", "up", "heavy"])
def test_golden_cases_bit_exact(tag):
    bits = GOLDEN[tag + "__w"]
    importance = GOLDEN[tag + "__importance"]
    offsets = tuple(int(o) for o in GOLDEN[tag + "__offsets"])
    w = dev(bits).view(torch.float16)
    q4, scales, stats = fp4_quant.quantize(w, dev(importance) if importance.size else None, offsets)
    assert (q4.cpu().numpy() == GOLDEN[tag + "__q4"]).all()
    assert (scales.cpu().numpy() == GOLDEN[tag + "__scales"]).all()
    assert stats["groups"] == scales.numel() and sum(stats["shift_groups"].values()) == scales.numel()
    assert stats["weighted_error_after"] <= stats["weighted_error_before"]
    np.testing.assert_allclose(stats["weighted_error_after"], GOLDEN[tag + "__error"].astype(np.float64).sum(), rtol=1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,k", [(1, 128), (129, 384), (1000, 3584)])
def test_random_matrices_match_the_oracle(dtype, rows, k):
    g = torch.Generator().manual_seed(SEED + rows)
    w = torch.randn(rows, k, generator=g) * 0.03
    w[torch.rand(rows, k, generator=g) < 0.01] *= 15
    w[0, :64] = 0
    w = w.to(dtype)
    importance = torch.rand(k, generator=g) * 3
    for weight, offsets in [(None, (0, -1, -2)), (importance, (0, -1, -2)), (importance, (0, 1, -1, -3))]:
        q4, scales, stats = fp4_quant.quantize(w.cuda(), None if weight is None else weight.cuda(), offsets)
        want_q4, want_scales = oracle.clip_pack(w, None if weight is None else weight.numpy(), offsets,
                                                bf16=dtype == torch.bfloat16)
        assert (scales.cpu().numpy() == want_scales).all()
        assert (q4.cpu().numpy() == want_q4).all()
        assert stats["shift_groups"]["0"] < scales.numel() or rows == 1


@pytest.mark.parametrize("weighted", [False, True])
def test_statistics_of_a_tall_matrix_do_not_drift(weighted):
    """One row repeated: the sums are the row's, times the number of rows, to the rounding of fp64 sums.  (20000 x 3584 gives a thread 59
    items; each item's fp32 part is the same in both calls, and a sum of N doubles is off by at most N 2^-53: 1e-9 for 9e6.)"""
    g = torch.Generator().manual_seed(SEED)
    rows, k = 20000, 3584
    row = (torch.randn(1, k, generator=g) * 0.03).bfloat16().cuda()
    importance = (torch.rand(k, generator=g) * 3).cuda() if weighted else None
    _, _, one = fp4_quant.quantize(row, importance)
    _, _, many = fp4_quant.quantize(row.expand(rows, k).contiguous(), importance)
    for name in ("weighted_error_before", "weighted_error_after", "weight_error_before", "weight_error_after"):
        assert abs(many[name] / (rows * one[name]) - 1) <= 1e-9, (name, many[name], rows * one[name])
    assert many["shift_groups"] == {s: rows * n for s, n in one["shift_groups"].items()}


def test_no_offsets_is_round_to_nearest_and_feeds_a_layer():
    """Without offsets the result is hg_pack's; a searched bank installs into a layer and changes only the low rows."""
    g = torch.Generator().manual_seed(SEED)
    w = (torch.randn(384, 512, generator=g) * 0.02).to(torch.bfloat16).cuda()
    q4, scales, _ = fp4_quant.quantize(w, offsets=())
    base_q, base_sf = native.pack(w, True)
    assert torch.equal(q4, base_q) and torch.equal(offline_weights.physical_scales(scales, 512), base_sf)
    ids = torch.arange(0, 384, 7, device="cuda")
    layer = native.DualLinear(w, ids)
    bank_q, bank_scales, stats = fp4_quant.quantize(w)
    offline_weights.replace_low_weight(layer, bank_q, bank_scales)
    x = torch.randn(8, 512, generator=g).to(torch.bfloat16).cuda()
    y = layer(x)
    dense = x.float() @ w.float().t()
    assert (y.float() - dense).norm() / dense.norm() < 0.12
    assert stats["weight_error_after"] <= stats["weight_error_before"]


@pytest.mark.parametrize("rows,k", [(1, 128), (7, 640), (9, 256), (1300, 3584)])
@pytest.mark.parametrize("kind", ["outstanding", "hidden", "signed", "missing"])
def test_candidates_ruled_out_by_one_term_never_win(rows, k, kind):
    """The plain entry point against the oracle, bit for bit, where the bound on a clipped candidate is tight, useless or not a bound:
    columns of outstanding importance, columns whose importance is zero (there the clipped candidate wins), negative and NaN importance."""
    g = torch.Generator().manual_seed(SEED + rows + k)
    w = torch.randn(rows, k, generator=g) * 0.03
    w[torch.rand(rows, k, generator=g) < 0.02] *= 8
    w = w.to(torch.bfloat16)
    importance = torch.rand(k, generator=g) + 0.1
    special = torch.rand(k, generator=g) < 0.05
    importance[special] = {"outstanding": 400.0, "hidden": 0.0, "signed": -2.0, "missing": float("nan")}[kind]
    if kind == "hidden":
        w[:, special] *= 8
    x, weight = w.cuda(), importance.cuda()
    for offsets in [(0, -1, -2), (-2, -1, 0), (-3, -2, -2, 1), (-1,), (-4, -8, 2, -2, 0, -1, 3, -3)]:
        q4 = torch.empty(rows, k // 2, dtype=torch.uint8, device="cuda")
        scales = torch.empty(rows, k // 32, dtype=torch.uint8, device="cuda")
        native.check(native.library().hg_clip_pack(x.data_ptr(), weight.data_ptr(), q4.data_ptr(), scales.data_ptr(), rows, k,
                                                   (native.C.c_int * len(offsets))(*offsets), len(offsets), 1,
                                                   native._stream(x.device)))
        want_q4, want_scales = oracle.clip_pack(w, importance.numpy(), offsets, bf16=True)
        assert (scales.cpu().numpy() == want_scales).all(), offsets
        assert (q4.cpu().numpy() == want_q4).all(), offsets


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["plain", "outstanding", "hidden"])
@pytest.mark.parametrize("rows,k", [(5, 128), (300, 640)])
def test_statistics_against_independent_sums(rows, k, kind, dtype):
    """How many groups moved by each offset, and the four error sums, against the oracle's codes.  All terms are non-negative; each is
    rounded three times in fp32 and eight are added in fp32 before fp64 takes over, so a sum is off by at most about 11 x 2^-24 = 7e-7."""
    g = torch.Generator().manual_seed(SEED + rows)
    w = torch.randn(rows, k, generator=g) * 0.03
    w[torch.rand(rows, k, generator=g) < 0.02] *= 8
    importance = torch.rand(k, generator=g) + 0.1
    special = torch.rand(k, generator=g) < 0.05
    if kind == "hidden":
        w[:, special] *= 8
    importance[special] = {"plain": 1.0, "outstanding": 400.0, "hidden": 0.0}[kind]
    w[0], w[1, :32], w[2, 32:64] = 0, 0, 1e-7
    w, weight = w.to(dtype), None if kind == "plain" else importance
    bf16, scale = dtype == torch.bfloat16, (torch.ones(k) if weight is None else weight).double()
    x = w.double()

    def error(packed, scale_bytes, per_column):
        values = fp4_quant.decode_logical(torch.from_numpy(packed), torch.from_numpy(scale_bytes), k).double()
        return float(((values - x).square() * per_column).sum())

    nearest = oracle.clip_pack(w, None, (), bf16=bf16)
    moves = set()
    for offsets in [(0, -1, -2), (-2, 3, -1, 0, 1), (2, -3, -4, -1, 0, 1, -2, -8), (-1,), ()]:
        q4, scales, stats = fp4_quant.quantize(w.cuda(), None if weight is None else weight.cuda(), offsets)
        want = oracle.clip_pack(w, None if weight is None else weight.numpy(), offsets, bf16=bf16)
        assert (scales.cpu().numpy() == want[1]).all() and (q4.cpu().numpy() == want[0]).all(), offsets
        moved = want[1].astype(np.int64) - nearest[1].astype(np.int64)
        assert stats["shift_groups"] == {str(-o): int((moved == o).sum()) for o in offsets}, offsets
        moves |= set(moved.ravel().tolist())
        for name, value in (("weighted_error_before", error(*nearest, scale)), ("weighted_error_after", error(*want, scale)),
                            ("weight_error_before", error(*nearest, 1.0)), ("weight_error_after", error(*want, 1.0))):
            np.testing.assert_allclose(stats[name], value, rtol=1e-6, err_msg=f"{name} {offsets}")
    assert moves >= ({0, -1} if kind != "hidden" else {0, -1, -2, -3})
