"""Gated Delta Net prefill on the GPU against the CPU oracle, the golden fixture of the
FlashInfer-Bench definition and the decode operator. Tolerances: fp32 recurrences in another
summation order (the state within 2e-5 of its largest value after hundreds of steps), bf16 outputs
within two rounding steps."""
import pytest
import torch

import oracle
from ako4x_b200 import _cabi, gdn_decode, gdn_prefill, workloads as W
from conftest import assert_close_bf16, load_golden

pytestmark = pytest.mark.gpu

KEYS = ("q", "k", "v", "state", "A_log", "a", "dt_bias", "b", "cu_seqlens")


def _run(a, scale="given"):
    args = [a[k].cuda() if a[k] is not None else None for k in KEYS]
    o, s = gdn_prefill.run(*args, a["scale"] if scale == "given" else scale)
    torch.cuda.synchronize()
    return o.cpu(), s.cpu()


def _check(o, s, ref_o, ref_s):
    assert o.shape == ref_o.shape and o.dtype == torch.bfloat16 and s.shape == ref_s.shape
    assert (s - ref_s).abs().max().item() <= 2e-5 * max(ref_s.abs().max().item(), 1e-3)
    assert_close_bf16(o, ref_o, atol=2e-3, rtol=2e-2)
    assert (o == ref_o).float().mean().item() > 0.9


def test_golden():
    g = load_golden("gdn_prefill_s3")
    a = W.make_gdn_prefill(g["inputs"]["seq_lens"], shape_id=g["inputs"]["shape_id"])
    o, s = _run(a)
    _check(o, s, g["outputs"]["output"], g["outputs"]["new_state"])
    assert torch.all(s[1] == 0)


@pytest.mark.parametrize("lens", [[1], [15], [16], [17], [33, 1, 64], [0, 100, 0, 7], [257]])
def test_against_oracle(lens):
    a = W.make_gdn_prefill(lens, shape_id=len(lens) + lens[0])
    o, s = _run(a)
    ro, rs = oracle.gdn_prefill(*[a[k] for k in KEYS], a["scale"])
    _check(o, s, ro, rs)


@pytest.mark.parametrize("lens", [[370], [33], [129], [16], [5], [70, 300], [0, 33], [17, 0]])
def test_both_forms_agree(lens):
    """Calls with a workspace run in the chunked form (32 tokens per step of the state) unless their sequences
    are a few tokens long; `_chunked=False` forces token by token. Both against the oracle and each other."""
    a = W.make_gdn_prefill(lens, shape_id=21 + len(lens))
    args = [a[k].cuda() if a[k] is not None else None for k in KEYS]
    o1, s1 = gdn_prefill.run(*args, a["scale"], _chunked=False)
    o2, s2 = gdn_prefill.run(*args, a["scale"])
    ro, rs = oracle.gdn_prefill(*[a[k] for k in KEYS], a["scale"])
    _check(o1.cpu(), s1.cpu(), ro, rs)
    _check(o2.cpu(), s2.cpu(), ro, rs)
    _check(o2.cpu(), s2.cpu(), o1.cpu(), s1.cpu())


def test_no_state_default_scale():
    a = W.make_gdn_prefill([40, 9], shape_id=5, with_state=False)
    o, s = _run(a, scale=None)
    ro, rs = oracle.gdn_prefill(*[a[k] for k in KEYS], None)
    _check(o, s, ro, rs)


def test_prefill_equals_repeated_decode():
    """A sequence run through prefill gives the outputs and the state of its tokens fed one by one
    through the decode operator (both on the GPU): 300 tokens, compared directly."""
    a = W.make_gdn_prefill([300], shape_id=11, device="cuda")
    o, s = gdn_prefill.run(*[a[k] for k in KEYS], a["scale"])
    st = a["state"]
    outs = []
    for t in range(300):
        ot, st = gdn_decode.run(a["q"][t:t + 1].unsqueeze(1), a["k"][t:t + 1].unsqueeze(1), a["v"][t:t + 1].unsqueeze(1),
                                st, a["A_log"], a["a"][t:t + 1].unsqueeze(1), a["dt_bias"], a["b"][t:t + 1].unsqueeze(1),
                                a["scale"])
        outs.append(ot[:, 0])
    od = torch.cat(outs)
    assert (s - st).abs().max().item() <= 2e-5 * st.abs().max().item()
    assert_close_bf16(o.cpu(), od.cpu(), atol=2e-3, rtol=2e-2)


def test_long_sequences_sampled():
    """8 192 tokens in four sequences (the largest recorded size): the last 64 outputs of one
    sequence and its final state against the oracle run on that sequence alone."""
    lens = [4096, 1024, 3000, 72]
    a = W.make_gdn_prefill(lens, shape_id=2, device="cuda")
    o, s = gdn_prefill.run(*[a[k] for k in KEYS], a["scale"])
    t0, t1 = 4096, 4096 + 1024
    one = {k: (a[k][t0:t1].cpu() if k in ("q", "k", "v", "a", "b") else a[k].cpu() if torch.is_tensor(a[k]) else a[k]) for k in KEYS}
    one["state"] = a["state"][1:2].cpu()
    one["cu_seqlens"] = torch.tensor([0, 1024])
    ro, rs = oracle.gdn_prefill(*[one[k] for k in KEYS], a["scale"])
    assert (s[1].cpu() - rs[0]).abs().max().item() <= 5e-5 * rs.abs().max().item()
    assert_close_bf16(o[t1 - 64:t1].cpu(), ro[-64:], atol=2e-3, rtol=2e-2)


@pytest.mark.parametrize("lens,lead,tail", [([31, 32, 33], 0, 0), ([1, 64, 0, 65, 2], 5, 9), ([96], 33, 1), ([0, 0, 7], 3, 0),
                                            ([40] * 70, 0, 40), ([31, 32, 33, 1, 0, 64, 65] * 3, 2, 3)])
def test_chunk_edges_and_tokens_outside(lens, lead, tail):
    """Sequences that end at, before and after a 32-token chunk, empty ones, more sequences than the
    slot search takes per step, and tokens in front of and behind every sequence (their outputs are
    zero). The chunked and the token-by-token form differ in the order of fp32 sums only: the state
    of n tokens within 2e-6 * sqrt(n) of its largest value."""
    a = W.make_gdn_prefill([lead] + lens + [tail], shape_id=31 + len(lens))
    n = len(lens)
    a["state"], a["cu_seqlens"] = a["state"][1:n + 1].contiguous(), a["cu_seqlens"][1:n + 2].contiguous()
    args = [a[k].cuda() for k in KEYS]
    o1, s1 = gdn_prefill.run(*args, a["scale"], _chunked=False)
    o2, s2 = gdn_prefill.run(*args, a["scale"])
    end = lead + sum(lens)
    assert torch.all(o2[:lead] == 0) and torch.all(o2[end:] == 0)
    assert (s1 - s2).abs().max().item() <= 2e-6 * max(lens) ** 0.5 * s1.abs().max().item()
    assert_close_bf16(o2.cpu(), o1.cpu(), atol=2e-3, rtol=2e-2)
    assert (o1 == o2).float().mean().item() > 0.99


@pytest.mark.parametrize("kind,value", [("v", "inf"), ("v", "nan"), ("k", "nan"), ("k", "-inf"), ("q", "nan"), ("a", "nan"),
                                        ("b", "nan"), ("a", "inf"), ("b", "-inf"), ("state", "nan"), ("state", "inf")])
@pytest.mark.parametrize("lens", [[75], [40, 7, 75], [75, 1, 40] + [5] * 21])
def test_values_that_are_not_finite_reach_no_earlier_token(kind, value, lens):
    """A value that is not finite spoils what the recurrence makes of it (its own output, or its row of the
    state from its token on) and nothing else: every other output and state element is as in the
    token-by-token form. Tokens at the edges and inside of the 8-, 16- and 32-token steps of the chunked
    form, and where there are several sequences the first one of another (the gate values +inf of `a` and
    -inf of `b` are zero decay and zero update: nothing is spoilt)."""
    a = W.make_gdn_prefill(lens, shape_id=77 + len(lens))
    start = 0 if lens[0] == 75 else lens[0] + lens[1]
    x = float(value)
    if kind == "state":
        a["state"][lens.index(75), 3, 17, 5] = x
        a["state"][lens.index(75), 6, 90, 127] = x
    else:
        t = {("v", "inf"): 20, ("v", "nan"): 63, ("k", "nan"): 9, ("k", "-inf"): 47, ("q", "nan"): 16, ("a", "nan"): 5,
             ("b", "nan"): 30, ("a", "inf"): 12, ("b", "-inf"): 55}[kind, value]
        a[kind][start + t].view(-1)[::3] = x
        if len(lens) > 1:
            a[kind][(start + 75) % sum(lens)].view(-1)[1] = x
    args = [a[k].cuda() for k in KEYS]
    o1, s1 = gdn_prefill.run(*args, a["scale"], _chunked=False)
    o2, s2 = gdn_prefill.run(*args, a["scale"])
    fo, fs = torch.isfinite(o1.float()), torch.isfinite(s1)
    assert torch.equal(torch.isfinite(o2.float()), fo) and torch.equal(torch.isfinite(s2), fs)
    if fs.any():
        assert (s1[fs] - s2[fs]).abs().max().item() <= 2e-6 * 75 ** 0.5 * s1[fs].abs().max().item()
    assert_close_bf16(o2[fo], o1[fo], atol=2e-3, rtol=2e-2)


@pytest.mark.parametrize("lens", [[1], [8], [1, 1, 1], [24, 0, 0], [0, 9, 15], [8] * 19, [1] * 18 + [134], [4] * 20, [2] * 63, [9], [25, 0, 0],
                                  [8] * 18 + [9], [4] * 19 + [5], [2] * 62 + [3], [1] * 64])
@pytest.mark.parametrize("state", [True, False])
def test_few_tokens_per_sequence(lens, state):
    """Sequences of a few tokens on average run token by token (up to 8 tokens for fewer than 20 sequences,
    4 for fewer than 32, 2 for fewer than 64), which is then the very same kernel; just above the line the
    two forms differ in the order of fp32 sums. Tokens in front of and behind the sequences are zero."""
    n = len(lens)
    most = n * (8 if n < 20 else 4 if n < 32 else 2 if n < 64 else 0)
    for lead, tail in ((0, 0), (2, 1)):
        a = W.make_gdn_prefill([lead] + lens + [tail], shape_id=13 + n, with_state=state)
        a["cu_seqlens"] = a["cu_seqlens"][1:n + 2].contiguous()
        if state:
            a["state"] = a["state"][1:n + 1].contiguous()
        args = [a[k].cuda() if a[k] is not None else None for k in KEYS]
        o1, s1 = gdn_prefill.run(*args, a["scale"], _chunked=False)
        o2, s2 = gdn_prefill.run(*args, a["scale"])
        assert torch.all(o2[:lead] == 0) and torch.all(o2[lead + sum(lens):] == 0)
        if lead + sum(lens) + tail <= most:
            assert torch.equal(o1, o2) and torch.equal(s1, s2)
        assert (s1 - s2).abs().max().item() <= 2e-6 * max(lens) ** 0.5 * max(s1.abs().max().item(), 1e-3)
        assert_close_bf16(o2.cpu(), o1.cpu(), atol=2e-3, rtol=2e-2)


@pytest.mark.parametrize("lens,offset,short,expected", [([40, 9, 50], 0, 16, 0), ([40, 9, 50], 8, 0, 0), ([40, 9, 50], 0, 0, 0),
                                                        ([40, 9], 0, 16, -4), ([40, 9], 8, 0, -4), ([40, 9], 0, 0, 0)])
def test_workspace_that_cannot_be_used(lens, offset, short, expected):
    """Too small (by `short` bytes) or misaligned: refused for one or two sequences, as good as none for more
    (the token-by-token form, whose outputs leave tokens outside the sequences as they are)."""
    L = _cabi.lib()
    a = W.make_gdn_prefill([3] + lens, shape_id=3, device="cuda")
    n, T = len(lens), 3 + sum(lens)
    a["state"], a["cu_seqlens"] = a["state"][1:].contiguous(), a["cu_seqlens"][1:].contiguous()
    need = L.ako4x_gdn_prefill_workspace_bytes(T, n)
    ws = torch.empty(need + 16, dtype=torch.uint8, device="cuda")
    o = torch.full((T, 8, 128), 7.0, dtype=torch.bfloat16, device="cuda")
    s = torch.empty((n, 8, 128, 128), device="cuda")
    st = L.ako4x_gdn_prefill(*[_cabi.ptr(a[k]) for k in KEYS], a["scale"], _cabi.ptr(o), _cabi.ptr(s), T, n,
                             ws.data_ptr() + offset, need - short, _cabi.stream())
    assert st == expected
    if expected == 0:
        ro, rs = gdn_prefill.run(*[a[k] for k in KEYS], a["scale"], _chunked=bool(not offset and not short))
        assert torch.equal(s, rs) and torch.equal(o[3:], ro[3:])
        assert torch.all(o[:3] == (7.0 if offset or short else 0.0))


@pytest.mark.parametrize("lens,state", [([300] * 8, True), ([700] * 2, False), ([100] * 24, True), ([900], True), ([50, 400, 33], True)])
@pytest.mark.parametrize("slow", [0, 5])
def test_state_precision(lens, state, slow):
    """The state's error from an fp64 recurrence is that of the token-by-token fp32 form: the chunked form has as
    many roundings of the values that matter, those of the tensor core twice as large (measured ratio of the rms
    errors 0.8 to 1.25; 2.2 to 3 where leading products were truncated more than once). `slow`: gates near 1,
    where errors add up over hundreds of tokens."""
    a = W.make_gdn_prefill(lens, shape_id=4, device="cuda", with_state=state)
    a["dt_bias"] = a["dt_bias"] - slow
    g = torch.exp(-torch.exp(a["A_log"].double()) * torch.nn.functional.softplus(a["a"].double() + a["dt_bias"].double()))
    beta, k, v = torch.sigmoid(a["b"].double()), a["k"].double().repeat_interleave(2, 1), a["v"].double()
    ref = torch.zeros(len(lens), 8, 128, 128, dtype=torch.float64, device="cuda") if not state else a["state"].double().clone()
    starts = a["cu_seqlens"].tolist()
    for t in range(max(lens)):
        on = torch.tensor([i for i, n in enumerate(lens) if t < n], device="cuda")
        pos = torch.tensor([starts[i] + t for i, n in enumerate(lens) if t < n], device="cuda")
        S = ref[on] * g[pos][..., None, None]
        delta = beta[pos][..., None] * (v[pos] - torch.einsum("nhvk,nhk->nhv", S, k[pos]))
        ref[on] = S + delta[..., None] * k[pos][:, :, None]
    args = [a[x] for x in KEYS]
    err = [(gdn_prefill.run(*args, a["scale"], _chunked=c)[1].double() - ref).norm().item() for c in (False, True)]
    assert err[1] <= 1.5 * err[0], err
