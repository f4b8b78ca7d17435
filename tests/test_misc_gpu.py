"""Sampling, gated-delta-net, conv, LoRA and MTP-glue kernels against their fp32 oracles."""
import pytest
import torch

from vllm_kunlun_b200 import ops
from vllm_kunlun_b200.ops.reference import basic as rb
from vllm_kunlun_b200.ops.reference import misc as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _surviving(logits, temperature, top_k, top_p):
    lg = logits.float() / temperature.unsqueeze(1)
    V = lg.shape[1]
    k = torch.where(top_k <= 0, torch.full_like(top_k, V), top_k)
    return ref.apply_top_k_top_p(lg.cpu(), k.cpu(), top_p.cpu()).softmax(-1)


@pytest.mark.parametrize("V", [1000, 151936])
def test_topk_topp_sample_matches_sort_based_masking(V):
    torch.manual_seed(0)
    B = 12
    logits = (torch.randn(B, V, device=DEV) * 3).to(torch.bfloat16)
    temp = torch.tensor([0.0, 1.0, 0.7, 1.3] * 3, device=DEV)
    top_k = torch.tensor([0, 0, 50, 5, 0, 1, 20, 0, 7, 0, 0, 100], dtype=torch.int32, device=DEV)
    top_p = torch.tensor([1.0, 0.9, 1.0, 0.5, 0.2, 1.0, 0.8, 1.0, 0.95, 0.05, 1.0, 0.6], device=DEV)
    noise = torch.empty(B, V, device=DEV).exponential_()
    got = ops.topk_topp_sample(logits, temp, top_k, top_p, noise=noise).cpu()
    t_safe = torch.where(temp == 0, torch.ones_like(temp), temp)
    probs = _surviving(logits, t_safe, top_k, top_p)
    want = (probs / noise.cpu()).argmax(-1)
    greedy = logits.float().argmax(-1).cpu()
    for b in range(B):
        if temp[b] == 0:
            assert got[b] == greedy[b]
        else:
            # the drawn token must be in the reference's surviving set; away from threshold ties it is the same token
            assert probs[b, got[b]] > 0, b
    same = (got == torch.where(temp.cpu() == 0, greedy, want)).float().mean()
    assert same >= 0.9
    # in-kernel generator: draws differ between calls and stay inside the surviving set
    a = ops.topk_topp_sample(logits, temp, top_k, top_p, seed=1).cpu()
    b2 = ops.topk_topp_sample(logits, temp, top_k, top_p, seed=1).cpu()
    for b in range(B):
        assert probs[b, a[b]] > 0 or temp[b] == 0
    assert (a != b2).any()


def test_sampling_distribution_is_unbiased():
    torch.manual_seed(1)
    V, n = 8, 4096
    row = torch.tensor([2.0, 1.0, 0.5, 0.0, -0.5, -1.0, -2.0, -3.0], device=DEV)
    logits = row.repeat(n, 1)
    temp = torch.ones(n, device=DEV)
    draws = ops.topk_topp_sample(logits, temp, None, None, seed=7).cpu()
    freq = torch.bincount(draws, minlength=V).float() / n
    torch.testing.assert_close(freq, row.softmax(-1).cpu(), atol=0.03, rtol=0)


def test_repetition_penalty():
    torch.manual_seed(2)
    B, V = 4, 5000
    logits = torch.randn(B, V, device=DEV)
    toks = torch.randint(0, V, (B, 64), device=DEV)
    toks[:, 10] = toks[:, 3]  # duplicates are penalised once
    n = torch.tensor([64, 10, 0, 33], dtype=torch.int32, device=DEV)
    pen = torch.tensor([1.2, 2.0, 1.5, 1.0], device=DEV)
    want = ops.apply_repetition_penalty(logits.cpu().clone(), toks.cpu(), n.cpu(), pen.cpu())
    got = ops.apply_repetition_penalty(logits.clone(), toks, n, pen)
    torch.testing.assert_close(got.cpu(), want)


def test_rejection_sample_kernel_matches_vectorised_reference():
    from vllm_kunlun_b200.sample.rejection_sampler import RejectionSampler
    torch.manual_seed(3)
    B, S, V = 6, 3, 2000
    num_draft = torch.tensor([3, 2, 0, 3, 1, 3], device=DEV)
    n = int(num_draft.sum())
    tp = torch.randn(n, V, device=DEV).softmax(-1)
    dp = torch.randn(n, V, device=DEV).softmax(-1)
    draft = tp.argmax(-1).clone()
    draft[1] = (draft[1] + 1) % V
    draft[4] = (draft[4] + 5) % V
    bonus = torch.randint(0, V, (B,), device=DEV)
    greedy = torch.tensor([True, False, True, False, True, False], device=DEV)
    u = torch.rand(n, device=DEV)
    rq = torch.empty(B, V, device=DEV).exponential_()
    for draft_probs in (dp, None):
        want = RejectionSampler().forward(draft, num_draft, tp, bonus, greedy, draft_probs, u, rq, S)
        got = ops.rejection_sample(draft, num_draft, tp, bonus, greedy, draft_probs, u, rq, S)
        assert torch.equal(got.cpu(), want.cpu())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_causal_conv1d_fn_and_update(dtype):
    torch.manual_seed(4)
    C, W, slots = 384, 4, 6
    cu = torch.tensor([0, 7, 7, 9, 40], dtype=torch.int32)
    T = int(cu[-1])
    x_wide = torch.randn(T, C + 64).to(dtype)
    x = x_wide[:, :C]  # a column slice of a wider projection
    w = (torch.randn(C, W) * 0.5).to(dtype)
    bias = torch.randn(C).to(dtype)
    states = torch.randn(slots, W - 1, C).to(dtype)
    idx = torch.tensor([3, 0, 5, 1], dtype=torch.int32)
    init = torch.tensor([1, 0, 0, 1], dtype=torch.int32)
    s_ref = states.clone()
    want = ref.causal_conv1d_fn(x, w, bias, cu, s_ref, idx, init, True)
    s_dev = states.to(DEV)
    got = ops.causal_conv1d_fn(x_wide.to(DEV)[:, :C], w.to(DEV), bias.to(DEV), cu.to(DEV), s_dev, idx.to(DEV), init.to(DEV), True)
    tol = dict(atol=2e-2, rtol=2e-2) if dtype == torch.bfloat16 else dict(atol=1e-5, rtol=1e-5)
    torch.testing.assert_close(got.cpu().float(), want.float(), **tol)
    torch.testing.assert_close(s_dev.cpu().float(), s_ref.float(), **tol)
    # decode step
    xb = torch.randn(4, C).to(dtype)
    idx2 = torch.tensor([3, -1, 5, 1], dtype=torch.int32)
    want2 = ref.causal_conv1d_update(xb, s_ref, w, bias, idx2, True)
    got2 = ops.causal_conv1d_update(xb.to(DEV), s_dev, w.to(DEV), bias.to(DEV), idx2.to(DEV), True)
    torch.testing.assert_close(got2.cpu().float(), want2.float(), **tol)
    torch.testing.assert_close(s_dev.cpu().float(), s_ref.float(), **tol)


@pytest.mark.parametrize("Dk,Dv,Hk,Hv", [(128, 128, 2, 4), (64, 32, 2, 2)])
def test_gated_delta_rule_varlen(Dk, Dv, Hk, Hv):
    torch.manual_seed(5)
    cu = torch.tensor([0, 1, 50, 50, 180], dtype=torch.int32)
    T = int(cu[-1])
    C = 2 * Hk * Dk + Hv * Dv
    mixed = torch.randn(T, C).to(torch.bfloat16)
    q = mixed[:, : Hk * Dk].view(T, Hk, Dk)
    k = mixed[:, Hk * Dk:2 * Hk * Dk].view(T, Hk, Dk)
    v = mixed[:, 2 * Hk * Dk:].view(T, Hv, Dv)
    A_log, dt_bias = torch.rand(Hv), torch.rand(Hv)
    a, b = torch.randn(T, Hv).to(torch.bfloat16), torch.randn(T, Hv).to(torch.bfloat16)
    g_ref, beta_ref = ops.fused_gdn_gating(A_log, a, b, dt_bias)
    g, beta = ops.fused_gdn_gating(A_log.to(DEV), a.to(DEV), b.to(DEV), dt_bias.to(DEV))
    torch.testing.assert_close(g.cpu(), g_ref, atol=1e-4, rtol=1e-4)
    torch.testing.assert_close(beta.cpu(), beta_ref, atol=1e-5, rtol=1e-5)
    states = torch.randn(5, Hv, Dv, Dk) * 0.1
    idx = torch.tensor([2, 0, 4, 1], dtype=torch.int32)
    init = torch.tensor([1, 1, 0, 0], dtype=torch.int32)
    s_ref = states.clone()
    want = ops.gated_delta_rule(q, k, v, g_ref, beta_ref, s_ref, cu, idx, init)
    s_dev = states.to(DEV)
    md = mixed.to(DEV)
    got = ops.gated_delta_rule(md[:, : Hk * Dk].view(T, Hk, Dk), md[:, Hk * Dk:2 * Hk * Dk].view(T, Hk, Dk),
                               md[:, 2 * Hk * Dk:].view(T, Hv, Dv), g, beta, s_dev, cu.to(DEV), idx.to(DEV), init.to(DEV))
    torch.testing.assert_close(got.cpu().float(), want.float(), atol=2e-2, rtol=2e-2)
    torch.testing.assert_close(s_dev.cpu(), s_ref, atol=2e-3, rtol=2e-3)


@pytest.mark.parametrize("lens,Hk,Hv,offset", [([1], 1, 1, 0), ([40], 1, 2, 0), ([64], 2, 2, 0), ([65, 0, 1, 63], 1, 2, 0),
                                               ([39, 128, 191, 7], 2, 4, 0), ([193, 16, 15, 40, 1], 16, 32, 0), ([130], 1, 2, 4)])
def test_gated_delta_rule_chunk_edges(lens, Hk, Hv, offset):
    """Requests around the lengths at which the chunk kernel takes over from the scan and around its chunks of 64 tokens, without
    rows, without a state slot, with and without a carried state; ``offset``: rows that no tensor map can read.  Both routes keep
    fp32 throughout: states agree to 2^-24 times the square root of the steps, with a factor of 30 for the sums of 128 terms and
    the state's cancellations (1e-4); outputs to the rounding of bf16 (2^-8 of the value) beside that."""
    torch.manual_seed(11)
    T, R, C = sum(lens), len(lens), (2 * Hk + Hv) * 128
    wide = torch.randn(T, C + 8).to(torch.bfloat16)
    g, beta = -torch.rand(T, Hv) * torch.tensor([0.02, 1.0])[torch.arange(Hv) % 2], torch.rand(T, Hv)
    states = torch.randn(R + 2, Hv, 128, 128) * 0.1
    slots = torch.randperm(R + 2)[:R].to(torch.int32)
    if R > 3:
        slots[-1] = -1
    init = (torch.arange(R) % 2).to(torch.int32)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)

    def run(dev):
        m, st = wide.to(dev)[:, offset:offset + C], states.to(dev)
        q, k, v = (m[:, a * 128:b * 128].view(T, b - a, 128) for a, b in ((0, Hk), (Hk, 2 * Hk), (2 * Hk, 2 * Hk + Hv)))
        return ops.gated_delta_rule(q, k, v, g.to(dev), beta.to(dev), st, cu.to(dev), slots.to(dev), init.to(dev)).cpu(), st.cpu()

    (got, got_st), (want, want_st) = run(DEV), run("cpu")
    torch.testing.assert_close(got_st, want_st, atol=1e-4, rtol=1e-4)
    n = T - (lens[-1] if R > 3 else 0)
    torch.testing.assert_close(got[:n].float(), want[:n].float(), atol=1e-3, rtol=2 ** -7)


@pytest.mark.parametrize("lens", [[4096], [2048, 1000, 3000]])
def test_gated_delta_rule_many_chunks(lens):
    """Up to 64 chunks a request: no wait gives up, and the results are the oracle's within the bounds given above."""
    from vllm_kunlun_b200.ops.gemm_cuda import check_status
    torch.manual_seed(21)
    T, R, Hk, Hv = sum(lens), len(lens), 1, 2
    q, k, v = (torch.randn(T, h, 128).bfloat16() for h in (Hk, Hk, Hv))
    g, beta = -torch.rand(T, Hv) * 0.05, torch.rand(T, Hv)
    slots, init = torch.arange(R).int(), torch.zeros(R).int()
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)

    def run(dev):
        st = torch.zeros(R, Hv, 128, 128, device=dev)
        return ops.gated_delta_rule(*(t.to(dev) for t in (q, k, v, g, beta)), st, cu.to(dev), slots.to(dev), init.to(dev)).cpu(), st.cpu()

    (got, got_st), (want, want_st) = run(DEV), run("cpu")
    check_status()
    torch.testing.assert_close(got_st, want_st, atol=1e-4, rtol=1e-4)
    torch.testing.assert_close(got.float(), want.float(), atol=1e-3, rtol=2 ** -7)


@pytest.mark.parametrize("bad", ["v", "k", "q", "g", "beta"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("at", [[77], [64], [0], [70, 71, 127, 200]])
def test_gated_delta_rule_bad_values_reach_later_tokens_only(bad, value, at):
    """A NaN or an infinity in tokens of the first of two requests: where the scan's outputs and states are finite the chunk form's
    are, and equal within the bounds given above; where the scan's are not, neither are they.  The other request, whose rows share
    a tile with the bad ones, keeps its bits, and so do tokens in front of the first bad one."""
    from vllm_kunlun_b200.ops.gemm_cuda import check_status
    torch.manual_seed(22)
    lens, Hk, Hv = [233, 90], 1, 2
    T = sum(lens)
    q, k, v = (torch.randn(T, h, 128).bfloat16() for h in (Hk, Hk, Hv))
    g, beta = -torch.rand(T, Hv) * 0.1, torch.rand(T, Hv)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    slots, init = torch.arange(2).int(), torch.ones(2).int()
    states = torch.randn(2, Hv, 128, 128) * 0.1

    def run(dev):
        st = states.to(dev)
        o = ops.gated_delta_rule(*(t.to(dev) for t in (q, k, v, g, beta)), st, cu.to(dev), slots.to(dev), init.to(dev))
        return o.cpu().float(), st.cpu()

    clean = run(DEV)
    t = dict(q=q, k=k, v=v, g=g, beta=beta)[bad]
    for i in at:
        t[i].view(-1)[1 if bad in ("g", "beta") else 5] = value
    got, want = run(DEV), run("cpu")
    check_status()
    assert torch.equal(got[0][:at[0]], clean[0][:at[0]])
    assert torch.equal(got[0][lens[0]:], clean[0][lens[0]:]) and torch.equal(got[1][1], clean[1][1])
    for a, b, tol in ((got[0], want[0], dict(atol=1e-3, rtol=2 ** -7)), (got[1], want[1], dict(atol=1e-4, rtol=1e-4))):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b))
        ok = torch.isfinite(b)
        torch.testing.assert_close(a[ok], b[ok], **tol)


@pytest.mark.parametrize("lens,Hk,Hv,Dv,dtype", [([1] * 5, 2, 4, 128, torch.bfloat16), ([2, 0, 1, 3], 1, 2, 64, torch.float16),
                                                 ([1, 1, 2], 2, 2, 32, torch.float32)])
@pytest.mark.parametrize("l2norm", [True, False])
def test_gated_delta_rule_steps(lens, Hk, Hv, Dv, dtype, l2norm):
    """A row or two a request (also none, and three): the decode kernel against the oracle.  Both in fp32 on the same inputs: states
    to 2^-24 times the 128 terms of a sum (1e-5), outputs to the rounding of their type beside that."""
    torch.manual_seed(12)
    T, R = sum(lens), len(lens)
    q, k, v = (torch.randn(T, h, d).mul(0.2).to(dtype) for h, d in ((Hk, 128), (Hk, 128), (Hv, Dv)))
    g, beta, states = -torch.rand(T, Hv), torch.rand(T, Hv), torch.randn(R + 1, Hv, Dv, 128) * 0.1
    slots, init = torch.randperm(R + 1)[:R].to(torch.int32), (torch.arange(R) % 2).to(torch.int32)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)

    def run(dev):
        st = states.to(dev)
        o = ops.gated_delta_rule(*(t.to(dev) for t in (q, k, v, g, beta)), st, cu.to(dev), slots.to(dev), init.to(dev), None, l2norm)
        return o.cpu().float(), st.cpu()

    (got, got_st), (want, want_st) = run(DEV), run("cpu")
    torch.testing.assert_close(got_st, want_st, atol=1e-5, rtol=1e-5)
    torch.testing.assert_close(got, want, atol=1e-5, rtol={torch.float32: 1e-4, torch.float16: 2 ** -9, torch.bfloat16: 2 ** -7}[dtype])


@pytest.mark.parametrize("lens,Hk,Hv", [([2] * 16, 2, 16), ([1] * 9 + [150], 8, 16), ([4, 1, 3], 1, 2), ([5, 1], 1, 2), ([16, 15, 1, 7], 16, 32),
                                        ([17, 1, 16], 16, 32), ([70] + [0] * 4, 2, 16)])
@pytest.mark.parametrize("host", ["exact", "none", "other"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gated_delta_rule_routes(lens, Hk, Hv, host, dtype):
    """Verification batches, mixed steps and lengths around the limits of the step kernel: the host's lengths choose kernels, and
    every length on the device has one that serves it, also where the host's are others (a captured step).  Bounds as above."""
    torch.manual_seed(23)
    T, R = sum(lens), len(lens)
    q, k, v = (torch.randn(T, h, 128).to(dtype) for h in (Hk, Hk, Hv))
    g, beta, states = -torch.rand(T, Hv) * 0.5, torch.rand(T, Hv), torch.randn(R + 1, Hv, 128, 128) * 0.1
    slots, init = torch.randperm(R + 1)[:R].to(torch.int32), (torch.arange(R) % 2).to(torch.int32)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    cu_host = dict(exact=cu.clone(), none=None, other=torch.arange(R + 1))[host]

    def run(dev):
        st = states.to(dev)
        o = ops.gated_delta_rule(*(t.to(dev) for t in (q, k, v, g, beta)), st, cu.to(dev), slots.to(dev), init.to(dev), None, True,
                                 cu_host if dev == DEV else None)
        return o.cpu().float(), st.cpu()

    (got, got_st), (want, want_st) = run(DEV), run("cpu")
    torch.testing.assert_close(got_st, want_st, atol=1e-4, rtol=1e-4)
    torch.testing.assert_close(got, want, atol=1e-3, rtol={torch.float32: 1e-4, torch.bfloat16: 2 ** -7}[dtype])


@pytest.mark.parametrize("W", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("lens", [[1] * 9, [7, 8, 9, 0, 1, 16], [515], [1] * 40 + [150, 3]])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_causal_conv1d_tokens_a_thread(W, lens, dtype):
    """Short requests and long ones, around the 8 and 16 tokens that a thread takes.  Sums of at most eight products in fp32 and a
    sigmoid to 2 units of 2^-23, rounded once to the type."""
    torch.manual_seed(24)
    T, R, ch = sum(lens), len(lens), 136
    x, w, st = torch.randn(T, ch).to(dtype), torch.randn(ch, W).to(dtype), torch.randn(R + 1, W - 1, ch).to(dtype)
    slots, init = torch.randperm(R + 1)[:R].to(torch.int32), (torch.arange(R) % 2).to(torch.int32)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    res = []
    for dev in (DEV, "cpu"):
        s = st.clone().to(dev)
        o = ops.causal_conv1d_fn(x.to(dev), w.to(dev), None, cu.to(dev), s, slots.to(dev), init.to(dev), True)
        res.append((o.cpu().float(), s.cpu()))
    torch.testing.assert_close(res[0][0], res[1][0], atol=1e-5, rtol=2 ** -7 if dtype == torch.bfloat16 else 1e-5)
    assert torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("flags", [torch.int32, torch.bool, torch.uint8, torch.int64])
@pytest.mark.parametrize("W", [2, 4, 9])
def test_single_token_convolution_and_flags(flags, W):
    """Per-request flags of every type that callers have, as the convolutions read them."""
    torch.manual_seed(19)
    R, ch = 5, 264
    x, w = torch.randn(R, ch).bfloat16(), torch.randn(ch, W).bfloat16()
    base = torch.randn(R + 1, W - 1, ch).bfloat16()
    slots, init = torch.tensor([3, 0, 4, 5, 1], dtype=torch.int32), torch.tensor([1, 0, 1, 1, 0]).to(flags)
    cu = torch.arange(R + 1, dtype=torch.int32)
    for one in (True, False):
        res = []
        for dev in (DEV, "cpu"):
            st = base.clone().to(dev)
            if one:
                o = ops.causal_conv1d_update(x.to(dev), st, w.to(dev), None, slots.to(dev), True, init.to(dev))
            else:
                o = ops.causal_conv1d_fn(x.to(dev), w.to(dev), None, cu.to(dev), st, slots.to(dev), init.to(dev), True)
            res.append((o.cpu().float(), st.cpu()))
        # fp32 sums of at most nine products, rounded to bf16 once: one step
        torch.testing.assert_close(res[0][0], res[1][0], rtol=2 ** -7, atol=1e-5)
        assert torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("rows", [[300, 0, 1, 63, 64, 65], [127, 128, 129, 257]])
@pytest.mark.parametrize("N,K,bias,pitch", [(512, 256, False, 520), (384, 128, True, 384), (200, 384, False, 216), (200, 384, True, 203)])
def test_grouped_fp8_wide_tiles(rows, N, K, bias, pitch):
    """128-row tiles of the fp8 grouped GEMM: empty, short and ragged groups, an odd number of weight blocks, rows that 16-byte stores
    cannot meet.  The products of a k-block are exact in 64 bits and summed in fp32 on the GPU: K / 128 + 128 roundings of 2^-24, far
    below the output's 2^-9, so the tolerance is that of bf16.  Nothing is written behind the last group's rows (an expert-parallel
    rank has more than its experts take), behind column N or in rows around the output."""
    from vllm_kunlun_b200.ops import _ext
    from vllm_kunlun_b200.ops.gemm_cuda import check_status
    torch.manual_seed(13)
    C, E, used = _ext.C(), len(rows), sum(rows)
    M = used + 150
    x = torch.randn(M, K, device=DEV).to(torch.float8_e4m3fn)
    w = torch.randn(E, N, K, device=DEV).to(torch.float8_e4m3fn)
    nb, kb = -(-N // 128), K // 128
    a_s, w_s = torch.rand(kb, (M + 3) // 4 * 4, device=DEV) + 0.1, torch.rand(E, nb, kb, device=DEV) + 0.1
    b = torch.randn(E, N, device=DEV).bfloat16() if bias else None
    lod = torch.tensor([0] + rows, device=DEV).cumsum(0).int()
    guarded = torch.full((M + 16, pitch), 12345.0, dtype=torch.bfloat16, device=DEV)
    out = guarded[8:8 + M, :N]
    C.grouped_gemm(out, x.view(torch.uint8), w.view(torch.uint8), lod, b, a_s, w_s, 128)
    check_status()
    want = torch.zeros(used, N, dtype=torch.float64, device=DEV)
    for e in range(E):
        r = slice(int(lod[e]), int(lod[e + 1]))
        for i in range(kb):
            c = slice(128 * i, 128 * i + 128)
            want[r] += (x[r, c].double() @ w[e, :, c].double().T) * a_s[i, r, None].double() * w_s[e, :, i].double().repeat_interleave(128)[:N]
        if bias:
            want[r] += b[e].double()
    torch.testing.assert_close(out[:used].double(), want, atol=1e-2, rtol=2 ** -8)
    guarded[8:8 + used, :N] = 12345.0
    assert bool((guarded == guarded[0, 0]).all())


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_grouped_fp8_with_activation(act, dtype):
    """Activation and quantiser in the epilogue of the first expert GEMM: the bytes and scales of the kernels that it replaces, and
    none behind the last group's rows."""
    from vllm_kunlun_b200.ops import _ext
    from vllm_kunlun_b200.ops.gemm_cuda import check_status
    torch.manual_seed(14)
    C, rows, inter, K = _ext.C(), [130, 1, 0, 64, 200], 256, 384
    E, used = len(rows), sum(rows)
    M = used + 133
    x = torch.randn(M, K, device=DEV).to(torch.float8_e4m3fn).view(torch.uint8)
    w = torch.randn(E, 2 * inter, K, device=DEV).to(torch.float8_e4m3fn).view(torch.uint8)
    a_s, w_s = torch.rand(K // 128, (M + 3) // 4 * 4, device=DEV) * 0.02, torch.rand(E, 2 * inter // 128, K // 128, device=DEV)
    b = torch.randn(E, 2 * inter, device=DEV).to(dtype)
    lod = torch.tensor([0] + rows, device=DEV).cumsum(0).int()
    h = torch.empty(M, 2 * inter, dtype=dtype, device=DEV)
    C.grouped_gemm(h, x, w, lod, b, a_s, w_s, 128)
    want_q, want_s = C.act_mul_quant_fp8(h, act, lod[E:])
    # the second call gets the first one's memory, which holds marks by then
    q, s = C.grouped_gemm_act_fp8(x, w, lod, b, a_s, w_s, act, h)
    at = q.data_ptr(), s.data_ptr()
    q.fill_(0xA5)
    s.fill_(-7.0)
    del q, s
    q, s = C.grouped_gemm_act_fp8(x, w, lod, b, a_s, w_s, act, h)
    check_status()
    assert torch.equal(q[:used], want_q[:used]) and torch.equal(s[:, :used], want_s[:, :used])
    assert (q.data_ptr(), s.data_ptr()) == at and bool((q[used:] == 0xA5).all()) and bool((s[:, used:] == -7.0).all())


@pytest.mark.parametrize("T,wide", [(2, False), (64, False), (300, True)])
def test_experts_ask_for_the_fused_epilogue_where_it_serves(T, wide, monkeypatch):
    """A decode batch does not pay for a call that turns it down."""
    from vllm_kunlun_b200.ops import _ext
    torch.manual_seed(25)
    C, E, H, inter, seen = _ext.C(), 8, 256, 128, []
    w13, w2 = (torch.randn(E, n, m, device=DEV).to(torch.float8_e4m3fn) for n, m in ((2 * inter, H), (H, inter)))
    s13, s2 = torch.rand(E, 2 * inter // 128, H // 128, device=DEV), torch.rand(E, H // 128, inter // 128, device=DEV)
    inner = C.grouped_gemm_act_fp8
    monkeypatch.setattr(C, "grouped_gemm_act_fp8", lambda *a: (seen.append(inner(*a)), seen[-1])[1])
    w, ids = ops.moe_route(torch.randn(T, E, device=DEV), 2, "softmax", True)
    ops.fused_moe(torch.randn(T, H, device=DEV).bfloat16(), w13, w2, w, ids, "silu", w13_scale=s13, w2_scale=s2)
    assert len(seen) == wide and all(seen)


@pytest.mark.parametrize("T,k,H,mapped", [(129, 8, 256, False), (300, 4, 2048 + 128, True)])
def test_moe_permute_quant(T, k, H, mapped):
    """Rows quantised on their way to their experts: every pair's row is the quantised row of its token, pairs of other ranks' experts
    have no place, and the places are those of the segments."""
    from vllm_kunlun_b200.ops import _ext
    torch.manual_seed(15)
    C, E = _ext.C(), 16
    x = torch.randn(T, H, device=DEV).bfloat16()
    ids = torch.rand(T, E, device=DEV).topk(k, -1).indices.int()
    emap = torch.where(torch.arange(E, device=DEV) % 2 == 0, torch.arange(E, device=DEV) // 2, -1).int() if mapped else None
    local = E // 2 if mapped else E
    q, st, pos, lod = C.moe_permute_quant(x, ids, emap, local, E, torch.zeros(2 * local, dtype=torch.int32, device=DEV))
    want_q, want_s = C.quant_fp8_group(x, False, None, 4)
    where = emap[ids.long()].flatten() if mapped else ids.flatten()
    assert torch.equal(pos < 0, where < 0)
    pair = (where >= 0).nonzero()[:, 0]
    p, token = pos[pair].long(), pair // k
    assert torch.equal(q[p], want_q[token]) and torch.equal(st[:, p], want_s[:, token])
    assert p.unique().numel() == pair.numel() == int(lod[-1])
    e = where[pair].long()
    assert bool(((p >= lod[e]) & (p < lod[e + 1])).all())


@pytest.mark.parametrize("T,Hq,Hkv,norm,dtype", [(1, 4, 2, True, torch.bfloat16), (257, 32, 8, False, torch.bfloat16),
                                                 (300, 5, 2, True, torch.float16), (40, 1, 1, False, torch.float16)])
@pytest.mark.parametrize("gemma", [False, True])
def test_qkv_rope_cache_wide_route(T, Hq, Hkv, norm, dtype, gemma):
    """Heads of 128 in 16-byte pieces against the general kernel, which the same rows take when they start off a 16-byte boundary:
    sums of 128 squares in another order, so that a value next to a rounding edge may move by one step of the 16-bit type."""
    from vllm_kunlun_b200.ops import _ext
    torch.manual_seed(16)
    C, width = _ext.C(), (Hq + 2 * Hkv) * 128
    buf = torch.randn(T, width + 8, device=DEV).to(dtype)
    w = [torch.randn(128, device=DEV).to(dtype) if norm else None for _ in range(2)]
    pos, slots = torch.randint(-1, 600, (T,), device=DEV), torch.randperm(512, device=DEV)[:T] - 3
    cos_sin = torch.randn(512, 128, device=DEV)
    res = []
    for off in (0, 1):
        rows = torch.empty(T, width + 8, dtype=dtype, device=DEV)[:, off:off + width]
        rows.copy_(buf[:, :width])
        q, cache = torch.zeros(T, Hq * 128, dtype=dtype, device=DEV), torch.zeros(8, 2, Hkv, 64, 128, dtype=dtype, device=DEV)
        C.qkv_split_norm_rope_cache(q, rows, pos, cos_sin, w[0], w[1], 1e-6, Hq, Hkv, 128, True, gemma, cache, slots)
        res.append((q.float(), cache.float()))
    step = 2 ** -7 if dtype == torch.bfloat16 else 2 ** -10
    for got, want in zip(*res):
        # two steps: one before the rotation, which mixes two columns, and one behind it
        torch.testing.assert_close(got, want, rtol=2 * step, atol=4 * step)
    if not norm:
        assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("rows", [1, 15, 16, 333])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_row_norms_of_128(rows, dtype, mode):
    """Rows of 128 in 16-byte pieces against the general kernel (the same rows off a 16-byte boundary): one rounding step apart."""
    from vllm_kunlun_b200.ops import _ext
    torch.manual_seed(17)
    x, z, w = (torch.randn(n, 128, device=DEV).to(dtype) for n in (rows, rows, 1))

    def run(off):
        def at(t):
            m = torch.empty(t.numel() + 8, dtype=dtype, device=DEV)[off:off + t.numel()].view(t.shape)
            return m.copy_(t)
        out = at(torch.zeros_like(x))
        _ext.C().rownorm(out, at(x), at(z) if mode >= 2 else None, None if mode == 1 else at(w)[0], 1e-6, mode)
        return out.float()

    torch.testing.assert_close(run(0), run(1), rtol=2 ** -7 if dtype == torch.bfloat16 else 2 ** -10, atol=1e-6)


@pytest.mark.parametrize("T,k,E,quant", [(1, 1, 8, True), (16, 8, 128, True), (33, 8, 512, False), (128, 8, 64, True), (300, 3, 16, False)])
@pytest.mark.parametrize("mapped", [False, True])
def test_moe_prepare_small_places(T, k, E, quant, mapped):
    """Places of a small batch's pairs: those of a stable sort by expert, rows and scales the token's."""
    from vllm_kunlun_b200.ops import _ext
    torch.manual_seed(18)
    C, H = _ext.C(), 384
    x = torch.randn(T, H, device=DEV).bfloat16()
    ids = torch.rand(T, E, device=DEV).topk(k, -1).indices.int()
    emap = torch.where(torch.arange(E, device=DEV) % 2 == 0, torch.arange(E, device=DEV) // 2, -1).int() if mapped else None
    local = E // 2 if mapped else E
    xs, pos, lod, st = C.moe_prepare_small(x, ids, emap, local, E, quant, None)
    where = (emap[ids.long()] if mapped else ids).flatten().long()
    order = torch.sort(torch.where(where < 0, local, where), stable=True).indices
    want = torch.empty_like(order)
    want[order] = torch.arange(T * k, device=DEV)
    assert torch.equal(pos.long(), torch.where(where < 0, -1, want))
    assert torch.equal(lod.long(), torch.searchsorted(torch.sort(where[where >= 0]).values, torch.arange(local + 1, device=DEV)))
    pair = (where >= 0).nonzero()[:, 0]
    p, token = pos[pair].long(), pair // k
    if quant:
        want_q, want_s = C.quant_fp8_group(x, False, None, 4)
        assert torch.equal(xs[p], want_q[token]) and torch.equal(st[:, p], want_s[:, token])
    else:
        assert torch.equal(xs[p], x[token])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("pattern", ["random", "segments"])
@pytest.mark.parametrize("N,offset,r", [(640, 128, 16), (333, 5, 8), (1030, 0, 12)])
def test_lora_shrink_expand(dtype, pattern, N, offset, r):
    """Token-tiled shrink / expand kernels vs the oracle: tiles whose tokens share an adapter (prefill segments), tiles
    with several adapters and base-model rows (-1), whole tiles of base-model rows, a token count off the tile sizes,
    odd column counts / offsets (no paired 4-byte stores), ranks that are not a multiple of the vector width,
    accumulate and overwrite."""
    torch.manual_seed(6)
    T, K, L = 77, 1024, 3
    x = torch.randn(T, K).to(dtype)
    A = (torch.randn(L, r, K) * 0.05).to(dtype)
    Bm = (torch.randn(L, N, r) * 0.05).to(dtype)
    if pattern == "random":
        ids = torch.randint(-1, L, (T,), dtype=torch.int32)
    else:   # runs of one adapter: 20 tokens of adapter 1, 20 base-model rows, 30 of adapter 0, 7 of adapter 2
        ids = torch.tensor([1] * 20 + [-1] * 20 + [0] * 30 + [2] * 7, dtype=torch.int32)
    h_ref = ref.bgmv_shrink(x, A, ids, 0.5)
    h = ops.lora_shrink(x.to(DEV), A.to(DEV), ids.to(DEV), 0.5)
    torch.testing.assert_close(h.cpu(), h_ref, atol=2e-3, rtol=2e-3)
    tol = dict(atol=3e-2, rtol=3e-2) if dtype == torch.bfloat16 else dict(atol=1e-4, rtol=1e-4)
    for add in (True, False):
        out0 = torch.randn(T, N + offset + 3).to(dtype)
        want = ref.bgmv_expand(h_ref, Bm, ids, out0.clone(), offset=offset, add=add)
        got = ops.lora_expand(h, Bm.to(DEV), ids.to(DEV), out0.to(DEV), offset=offset, add=add)
        torch.testing.assert_close(got.cpu().float(), want.float(), **tol)


def test_mtp_concat_norm_and_sigmoid_gate():
    torch.manual_seed(7)
    T, H = 9, 1024
    e, h = torch.randn(T, H).to(torch.bfloat16), torch.randn(T, H).to(torch.bfloat16)
    we, wh = torch.rand(H).to(torch.bfloat16), torch.rand(H).to(torch.bfloat16)
    pos = torch.tensor([0, 1, 2, 0, 5, 6, 7, 0, 1])
    want = ops.mtp_concat_norm(e, h, we, wh, 1e-6, pos)
    got = ops.mtp_concat_norm(e.to(DEV), h.to(DEV), we.to(DEV), wh.to(DEV), 1e-6, pos.to(DEV))
    torch.testing.assert_close(got.cpu().float(), want.float(), atol=2e-2, rtol=2e-2)
    wide = torch.randn(T, 3 * H).to(torch.bfloat16)
    o = torch.randn(T, H).to(torch.bfloat16)
    want = ops.sigmoid_gate_mul(o, wide[:, :H])
    got = ops.sigmoid_gate_mul(o.to(DEV), wide.to(DEV)[:, :H])
    torch.testing.assert_close(got.cpu().float(), want.float(), atol=2e-2, rtol=2e-2)


def _first_logits(llm, prompt):
    from vllm_kunlun_b200 import SamplingParams
    from vllm_kunlun_b200.attention.metadata import ForwardContext, set_forward_context
    eng = llm.engine
    eng.add_request(prompt, SamplingParams(max_tokens=1))
    sched = eng.scheduler.schedule()
    md, ids, _ = eng.runner.prepare(sched)
    lora = None if eng.runner.lora is None else eng.runner.lora.punica
    with torch.inference_mode(), set_forward_context(ForwardContext(md, eng.runner.kv_caches, eng.pstate, lora=lora)):
        h, _ = eng.runner.model(ids)
        return eng.runner.model.compute_logits(h[-1:]).float().cpu()


def test_hybrid_engine_on_gpu():
    import dataclasses

    from vllm_kunlun_b200 import LLM, SamplingParams
    from vllm_kunlun_b200.config import qwen3_next_80b_a3b, tiny
    cfg = tiny(qwen3_next_80b_a3b(), num_layers=4, vocab_size=2048, hidden_size=512, num_heads=8, num_kv_heads=2,
               head_dim=64, rotary_dim=16, intermediate_size=512, num_experts=4, num_experts_per_tok=4,  # no routing ties
               moe_intermediate_size=256, gdn_num_k_heads=2, gdn_num_v_heads=4, gdn_head_k_dim=64, gdn_head_v_dim=64,
               max_position=1024)
    kw = dict(block_size=16, max_model_len=512, max_num_seqs=4, num_gpu_blocks=128, max_num_batched_tokens=256)
    gpu = LLM(cfg, device="cuda", enforce_eager=True, **kw)
    cpu = LLM(dataclasses.replace(cfg, dtype="float32"), device="cpu", **kw)
    sd = {k: v.float().cpu() for k, v in gpu.engine.runner.model.state_dict().items()}
    with torch.inference_mode():
        cpu.engine.runner.model.load_state_dict(sd)
    prompt = torch.randint(0, 2048, (150,), generator=torch.Generator().manual_seed(0)).tolist()
    cos = torch.nn.functional.cosine_similarity(_first_logits(gpu, prompt), _first_logits(cpu, prompt)).item()
    assert cos > 0.99, cos
    prompts = [list(range(3, 70)), list(range(100, 117)), list(range(200, 203))]
    sp = SamplingParams(max_tokens=12, ignore_eos=True)
    outs = []
    for eager in (True, False):
        llm = LLM(cfg, device="cuda", enforce_eager=eager, seed=5, **kw)
        outs.append([o.token_ids for o in llm.generate(prompts, sp)])
    assert outs[0] == outs[1]


def test_lora_engine_on_gpu():
    import dataclasses

    from test_lora_cpu import _adapter, _cfg
    from vllm_kunlun_b200 import LLM, SamplingParams
    cfg = dataclasses.replace(_cfg(512, 8, 2, 64, 1024, 2048), dtype="bfloat16")
    kw = dict(block_size=16, max_model_len=128, max_num_seqs=4, num_gpu_blocks=32, enable_lora=True, max_loras=2,
              max_lora_rank=8)
    reqs = [_adapter(cfg, 1), _adapter(cfg, 2, r=8, alpha=4.0, targets=("k_proj", "up_proj", "o_proj")), None]
    gpu = LLM(cfg, device="cuda", enforce_eager=True, **kw)
    cpu = LLM(dataclasses.replace(cfg, dtype="float32"), device="cpu", **kw)
    sd = {k: v.float().cpu() for k, v in gpu.engine.runner.model.state_dict().items()}
    with torch.inference_mode():
        cpu.engine.runner.model.load_state_dict(sd)
    for llm in (gpu, cpu):
        llm.add_lora(reqs[0])
    prompt = list(range(3, 60))
    for llm in (gpu, cpu):
        llm.engine.add_request([1, 2, 3], SamplingParams(max_tokens=1), lora_id=-1)  # a base-model row in the same step
    a, b = [], []
    for llm, dst in ((gpu, a), (cpu, b)):
        eng = llm.engine
        eng.add_request(prompt, SamplingParams(max_tokens=1), lora_id=1)
        sched = eng.scheduler.schedule()
        md, ids, _ = eng.runner.prepare(sched)
        from vllm_kunlun_b200.attention.metadata import ForwardContext, set_forward_context
        with torch.inference_mode(), set_forward_context(
                ForwardContext(md, eng.runner.kv_caches, eng.pstate, lora=eng.runner.lora.punica)):
            h, _ = eng.runner.model(ids)
            dst.append(eng.runner.model.compute_logits(h[-1:]).float().cpu())
    cos = torch.nn.functional.cosine_similarity(a[0], b[0]).item()
    assert cos > 0.99, cos
    prompts = [list(range(3, 20)), list(range(30, 41)), list(range(50, 58))]
    sp = SamplingParams(max_tokens=6, ignore_eos=True)
    outs = []
    for eager in (True, False):
        llm = LLM(cfg, device="cuda", enforce_eager=eager, seed=2, **kw)
        outs.append([o.token_ids for o in llm.generate(prompts, sp, lora_request=reqs)])
    assert outs[0] == outs[1]
    base = LLM(cfg, device="cuda", enforce_eager=True, seed=2, **{k: v for k, v in kw.items() if "lora" not in k})
    assert [o.token_ids for o in base.generate(prompts[2:], sp)] == outs[0][2:]


@pytest.mark.parametrize("D", [64, 80, 128])
def test_varlen_bidirectional_attention(D):
    torch.manual_seed(8)
    H = 4
    cu = torch.tensor([0, 100, 100, 357, 400], dtype=torch.int32)
    T = int(cu[-1])
    q, k, v = (torch.randn(T, H, D).to(torch.bfloat16) for _ in range(3))
    want = ops.varlen_attention(q, k, v, cu)
    got = ops.varlen_attention(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV))
    torch.testing.assert_close(got.cpu().float(), want.float(), atol=2e-2, rtol=2e-2)


def test_qwen_vl_engine_on_gpu():
    import dataclasses

    from test_vision_cpu import IMG, _qwen_vl
    from vllm_kunlun_b200 import LLM, SamplingParams
    cfg = _qwen_vl()
    cfg = dataclasses.replace(cfg, hidden_size=512, num_heads=8, num_kv_heads=2, head_dim=64, v_head_dim=64, rotary_dim=64,
                              intermediate_size=1024, vocab_size=2048, dtype="bfloat16", mrope_section=(8, 12, 12))
    cfg.vision = dict(cfg.vision, hidden=128, heads=2, intermediate=256, patch=4, image_token_id=2047)
    grid = [(1, 16, 8)]
    px = torch.randn(128, 3 * 1 * 4 * 4, generator=torch.Generator().manual_seed(0))
    prompt = [5, 6, 7] + [2047] * 32 + [9, 10, 11, 12]
    kw = dict(block_size=16, max_model_len=256, max_num_seqs=4, num_gpu_blocks=64)
    gpu = LLM(cfg, device="cuda", enforce_eager=True, **kw)
    cpu = LLM(dataclasses.replace(cfg, dtype="float32"), device="cpu", **kw)
    sd = {k: v.float().cpu() for k, v in gpu.engine.runner.model.state_dict().items()}
    with torch.inference_mode():
        cpu.engine.runner.model.load_state_dict(sd)
    mm = {"pixel_values": px, "image_grid_thw": grid}
    ea = gpu.engine.runner.model.embed_multimodal(px, grid).float().cpu()
    eb = cpu.engine.runner.model.embed_multimodal(px, grid).float()
    assert torch.nn.functional.cosine_similarity(ea.flatten(), eb.flatten(), dim=0) > 0.99

    def logits(llm):
        from vllm_kunlun_b200.attention.metadata import ForwardContext, set_forward_context
        eng = llm.engine
        eng.add_request(prompt, SamplingParams(max_tokens=1), multi_modal_data=mm)
        sched = eng.scheduler.schedule()
        md, ids, _ = eng.runner.prepare(sched)
        ctx = ForwardContext(md, eng.runner.kv_caches, eng.pstate, extras=eng.runner._step_extras)
        with torch.inference_mode(), set_forward_context(ctx):
            h, _ = eng.runner.model(ids)
            return eng.runner.model.compute_logits(h[-1:]).float().cpu()

    cos = torch.nn.functional.cosine_similarity(logits(gpu), logits(cpu)).item()
    assert cos > 0.99, cos
    out = LLM(cfg, device="cuda", **kw).generate([prompt], SamplingParams(max_tokens=5, ignore_eos=True), multi_modal_data=mm)
    assert len(out[0].token_ids) == 5

