"""Paged GQA decode parity through the C ABI."""
import pytest
import torch

import oracle
from ako4x_b200 import _cabi, gqa_decode, workloads as W
from conftest import assert_close_bf16, assert_lse_close, load_golden

pytestmark = pytest.mark.gpu
KEYS = ["q", "k_cache", "v_cache", "kv_indptr", "kv_indices", "sm_scale"]


def _run(a):
    d = W.to_device(a, "cuda")
    return gqa_decode.run(*[d[k] for k in KEYS])


def _check(a):
    o, lse = _run(a)
    ro, rlse = oracle.gqa_paged_decode(*[a[k] for k in KEYS])
    assert_close_bf16(o, ro)
    assert_lse_close(lse, rlse)


def test_golden(built_lib):
    g = load_golden("gqa_decode_b4")
    o, lse = _run(g["inputs"])
    assert_close_bf16(o, g["outputs"]["output"])
    assert_lse_close(lse, g["outputs"]["lse"])


@pytest.mark.parametrize("lens", [[1], [15], [16], [17], [128], [547], [2100],
                                  [0, 1, 0], [40, 0, 300, 7, 1024], [8192]])
def test_ragged_lengths(built_lib, lens):
    _check(W.make_gqa_decode(len(lens), shape_id=sum(lens) % 89, lens=lens, extra_pages=13))


@pytest.mark.parametrize("batch", [1, 16, 64])
def test_config_shapes(built_lib, batch):
    """Benchmark configuration shapes, with lengths capped so the CPU oracle stays fast."""
    _check(W.make_gqa_decode(batch, shape_id=batch, len_lo=128, len_hi=1024 if batch > 1 else 8192))


def test_work_list_mode_ragged(built_lib):
    """Very long next to very short and empty sequences, cut into equal shares, checked against the oracle for
    every row."""
    lens = [8192] * 20 + [1, 17, 300, 0, 2049, 255, 256, 257] + [5000, 16, 0, 777] * 5
    assert sum(lens) >= 160 * 1024
    _check(W.make_gqa_decode(len(lens), shape_id=41, lens=lens, extra_pages=29))


def test_page_size_4(built_lib):
    g = torch.Generator().manual_seed(5)
    pages, P = 50, 4
    q = torch.randn(2, 32, 128, generator=g).to(torch.bfloat16)
    k = torch.randn(pages, P, 8, 128, generator=g).to(torch.bfloat16)
    v = torch.randn(pages, P, 8, 128, generator=g).to(torch.bfloat16)
    indptr = torch.tensor([0, 7, 19], dtype=torch.int32)
    idx = torch.randperm(pages, generator=g)[:19].to(torch.int32)
    a = dict(q=q, k_cache=k, v_cache=v, kv_indptr=indptr, kv_indices=idx, sm_scale=0.09)
    _check(a)


def test_full_size_split_invariance(built_lib):
    """B=256 at full lengths: appending a key with logit -> -inf weight changes nothing, and
    lse matches a direct fp32 recomputation on one sampled sequence."""
    a = W.make_gqa_decode(256, shape_id=3, device="cuda")
    o, lse = gqa_decode.run(*[a[k] for k in KEYS])
    assert torch.isfinite(o.float()).all() and torch.isfinite(lse).all()
    b = 37
    s, e = int(a["kv_indptr"][b]), int(a["kv_indptr"][b + 1])
    rows = a["kv_indices"][s:e].long()
    k = a["k_cache"][rows, 0].float()            # [L, 8, 128]
    v = a["v_cache"][rows, 0].float()
    qb = a["q"][b].float().view(8, 4, 128)
    logits = torch.einsum("hgd,lhd->hgl", qb, k) * a["sm_scale"]
    ref_lse = (torch.logsumexp(logits, -1) / 0.6931471805599453).reshape(32)
    ref_o = torch.einsum("hgl,lhd->hgd", torch.softmax(logits, -1), v).reshape(32, 128)
    assert_lse_close(lse[b], ref_lse)
    assert_close_bf16(o[b], ref_o.to(torch.bfloat16))


def test_full_length_sampled_sequences(built_lib):
    """B = 256 with the configured lengths (128..8192): eight sampled sequences against the CPU oracle
    (their cache rows compacted into a small cache)."""
    a = W.make_gqa_decode(256, shape_id=256, device="cuda")
    o, lse = gqa_decode.run(*[a[k] for k in KEYS])
    sel = [0, 1, 50, 99, 128, 200, 254, 255]
    ip = a["kv_indptr"].cpu().long()
    rows, indptr = [], [0]
    for b in sel:
        rows.append(a["kv_indices"][ip[b]:ip[b + 1]].long())
        indptr.append(indptr[-1] + int(ip[b + 1] - ip[b]))
    rows = torch.cat(rows)
    dsel = torch.tensor(sel, device="cuda")
    ro, rlse = oracle.gqa_paged_decode(a["q"][dsel].cpu(), a["k_cache"][rows].cpu(), a["v_cache"][rows].cpu(),
                                       torch.tensor(indptr, dtype=torch.int32),
                                       torch.arange(rows.numel(), dtype=torch.int32), a["sm_scale"])
    assert_close_bf16(o[dsel], ro)
    assert_lse_close(lse[dsel], rlse)


def test_non_contiguous_query(built_lib):
    """q as a strided view: the wrapper's contiguous copy must be alive when the kernel runs."""
    a = W.make_gqa_decode(3, shape_id=17, lens=[300, 1, 2049], extra_pages=7)
    d = W.to_device(a, "cuda")
    wide = torch.zeros((3, 32, 256), dtype=torch.bfloat16, device="cuda")
    wide[..., :128] = d["q"]
    o, lse = gqa_decode.run(wide[..., :128], *[d[k] for k in KEYS[1:]])
    ro, rlse = oracle.gqa_paged_decode(*[a[k] for k in KEYS])
    assert_close_bf16(o, ro)
    assert_lse_close(lse, rlse)


def test_same_buffers_new_contents(built_lib):
    a = W.to_device(W.make_gqa_decode(3, lens=[70, 300, 5], extra_pages=3), "cuda")
    o1, _ = gqa_decode.run(*[a[k] for k in KEYS])
    o1 = o1.clone()
    a["v_cache"].mul_(-1)
    o2, _ = gqa_decode.run(*[a[k] for k in KEYS])
    assert torch.equal(o2, -o1)


@pytest.mark.parametrize("lens", [[15, 16, 17, 0, 33, 1] * 40, [600] * 3 + [0] + [3] * 230, [5, 0, 8192, 2, 0], [7000, 16, 1]])
def test_shares_and_whole_sequences(built_lib, lens):
    """Many short sequences, most of them inside one share, some longer ones among them, and few sequences whose
    partials come from one or from hundreds of shares; empty ones in between."""
    _check(W.make_gqa_decode(len(lens), shape_id=60 + len(lens) % 7, lens=lens, extra_pages=11))


@pytest.mark.parametrize("lens", [[1], [5], [8, 9], [21, 16, 47], [700, 30], [7] * 230])
def test_infinity_in_the_last_value_row(built_lib, lens):
    """The lanes of a last tile that have no token of their own read the last one again, with weight 0: an
    infinity there stays one (0 x inf would make it NaN)."""
    a = W.make_gqa_decode(len(lens), shape_id=5, lens=lens, extra_pages=3)
    for b in range(len(lens)):
        a["v_cache"][int(a["kv_indices"][int(a["kv_indptr"][b + 1]) - 1]), 0, b % 8, 40 + b % 64] = float("inf") if b % 2 else float("-inf")
    o, lse = _run(a)
    ro, rlse = oracle.gqa_paged_decode(*[a[k] for k in KEYS])
    assert torch.equal(o.cpu()[~torch.isfinite(ro)], ro[~torch.isfinite(ro)]) and torch.isfinite(o.cpu()[torch.isfinite(ro)]).all()
    assert torch.isinf(ro).any() and not torch.isnan(ro).any()
    assert_close_bf16(o.cpu()[torch.isfinite(ro)], ro[torch.isfinite(ro)])
    assert_lse_close(lse, rlse)


@pytest.mark.parametrize("length,masked", [(64, range(0, 32)), (64, range(32, 64)), (2100, range(0, 700)), (2100, range(900, 2100)), (40, range(0, 39)),
                                           (3000, range(16, 32))])
def test_keys_that_score_minus_infinity(built_lib, length, masked):
    """Keys whose dot product overflows to -inf weigh nothing, also where they fill whole tiles and shares."""
    a = W.make_gqa_decode(2, shape_id=9, lens=[length, 50], extra_pages=3)
    a["q"] = a["q"].abs() + 1e3
    rows = a["kv_indices"][:length][torch.tensor(list(masked))].long()
    a["k_cache"] *= 1e-3
    a["k_cache"][rows] = -3e38
    o, lse = _run(a)
    ro, rlse = oracle.gqa_paged_decode(*[a[k] for k in KEYS])
    assert torch.isfinite(ro.float()).all() and torch.isfinite(o.float()).all()
    assert_close_bf16(o, ro)
    assert_lse_close(lse, rlse)


@pytest.mark.parametrize("lens", [[512] * 222, [513] * 222, [512] * 221, [100] * 221 + [4000, 3], [3000] + [0, 17] * 130, [0, 31, 5] * 300 + [2500],
                                  [16] * 889, [6000, 0, 0] + [1] * 250 + [0] * 40 + [700, 650]])
def test_large_batches_with_and_without_a_workspace(built_lib, lens):
    """Batches on both sides of what is accepted without a workspace (mean length 512 from 222 sequences on,
    any from 888 on, on 148 SMs), some with one sequence far longer than the rest: cut at share boundaries with
    one merge entry per share, and whole sequences per CTA pair, against the oracle and each other."""
    a = W.make_gqa_decode(len(lens), shape_id=3, lens=lens, extra_pages=5)
    _check(a)
    d = W.to_device(a, "cuda")
    L, n, idx = _cabi.lib(), len(lens), a["kv_indices"].numel()
    o, lse = torch.full_like(d["q"], float("nan")), torch.full((n, 32), float("nan"), device="cuda")
    st = L.ako4x_gqa_paged_decode(*[_cabi.ptr(d[k]) for k in KEYS[:5]], d["sm_scale"], _cabi.ptr(o), _cabi.ptr(lse), n, idx, 1, None, 0,
                                  _cabi.stream())
    without = n >= 888 or (n >= 222 and idx <= 512 * n)
    assert st == (0 if without else -4)
    if without:
        ro, rlse = gqa_decode.run(*[d[k] for k in KEYS])
        assert_close_bf16(o, ro)
        assert_lse_close(lse, rlse)


def test_a_long_sequence_in_a_large_batch_is_shared(built_lib):
    """256 sequences with a mean below 512 tokens, one of which holds half of the tokens: it must not be left to
    one pair of CTAs, which takes more than ten times as long as a batch of equal sequences of the same size."""
    def us(lens):
        a = W.make_gqa_decode(len(lens), shape_id=1, lens=lens, device="cuda", extra_pages=3)
        args = [a[k] for k in KEYS]
        best = 1e9
        for _ in range(5):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            gqa_decode.run(*args)
            ev[1].record()
            torch.cuda.synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]) * 1e3)
        return best
    assert us([32768] + [128] * 255) < 3 * us([256] * 256)


@pytest.mark.parametrize("lens", [[547], [8192], [4000, 300, 7000] * 10, [700] * 230])
def test_precision_is_that_of_the_output(built_lib, lens):
    """Relative Frobenius error from an fp64 result: rounding the output to bf16 alone leaves 1.66e-3 (uniform
    rounding errors of at most 2^-9 over a binade), 16-bit weights and fp32 sums add less than 1e-5 to it."""
    a = W.make_gqa_decode(len(lens), shape_id=8, lens=lens, device="cuda", extra_pages=3)
    o, lse = gqa_decode.run(*[a[k] for k in KEYS])
    ref = []
    for b in range(len(lens)):
        rows = a["kv_indices"][int(a["kv_indptr"][b]):int(a["kv_indptr"][b + 1])].long()
        s = torch.einsum("hgd,lhd->hgl", a["q"][b].double().view(8, 4, 128), a["k_cache"][rows, 0].double()) * a["sm_scale"]
        ref.append(torch.einsum("hgl,lhd->hgd", s.softmax(-1), a["v_cache"][rows, 0].double()).reshape(32, 128))
    ref = torch.stack(ref)
    assert ((o.double() - ref).norm() / ref.norm()).item() < 1.75e-3
