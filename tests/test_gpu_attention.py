"""tcgen05 flash attention (forward and backward) against the fp32 PyTorch restatement."""
import math

import pytest
import torch

from picotron_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    from picotron_b200.ops import _ext
    return _ext.load()


def rnd(*shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


CASES = [
    # B, Sq, Sk, hq, hkv, d, causal
    (2, 256, 256, 4, 2, 64, True),
    (1, 128, 128, 2, 2, 64, True),
    (2, 300, 300, 4, 4, 64, True),      # ragged tail
    (1, 1024, 1024, 4, 1, 64, True),
    (1, 16, 16, 2, 1, 64, True),        # tiny (the multi-GPU tests use such sizes)
    (2, 256, 256, 2, 1, 128, True),
    (1, 200, 200, 2, 2, 128, True),
    (1, 128, 384, 4, 2, 64, False),     # full attention, Sq != Sk (ring blocks from earlier ranks)
    (1, 200, 136, 2, 2, 128, False),
]


@pytest.mark.parametrize("B,Sq,Sk,hq,hkv,d,causal", CASES)
def test_attention_forward(C, B, Sq, Sk, hq, hkv, d, causal):
    q, k, v = rnd(B, Sq, hq, d, seed=1), rnd(B, Sk, hkv, d, seed=2), rnd(B, Sk, hkv, d, seed=3)
    scale = 1.0 / math.sqrt(d)
    o, lse = C.attention_fwd(q, k, v, causal, scale)
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    o_ref, lse_ref = ref.attention_fwd(q, k, v, causal, scale)
    torch.testing.assert_close(lse, lse_ref, rtol=1e-3, atol=2e-3)
    torch.testing.assert_close(o.float(), o_ref.float(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("B,Sq,Sk,hq,hkv,d,causal", CASES)
def test_attention_backward(C, B, Sq, Sk, hq, hkv, d, causal):
    q, k, v = rnd(B, Sq, hq, d, seed=1), rnd(B, Sk, hkv, d, seed=2), rnd(B, Sk, hkv, d, seed=3)
    do = rnd(B, Sq, hq, d, seed=4)
    scale = 1.0 / math.sqrt(d)
    o_ref, lse_ref = ref.attention_fwd(q, k, v, causal, scale)
    dq_r, dk_r, dv_r = ref.attention_bwd(do, q, k, v, o_ref, lse_ref, causal, scale)
    dq, dk, dv = C.attention_bwd(do, q, k, v, o_ref, lse_ref, causal, scale)
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    for name, got, want in (("dq", dq, dq_r), ("dk", dk, dk_r), ("dv", dv, dv_r)):
        err = float((got.float() - want).norm() / (want.norm() + 1e-12))
        assert err < 2e-2, f"{name}: relative error {err:.4f}"
        torch.testing.assert_close(got.float(), want, rtol=5e-2, atol=5e-2)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("Sq,Sk,causal", [(517, 517, True), (300, 517, False), (129, 640, False)])
@pytest.mark.parametrize("rows", ["all", "some", "none"])
def test_attention_forward_moves_its_reference_maximum(C, Sq, Sk, causal, d, rows):
    """Keys that grow with every 64, so that a row's maximum jumps by far more than the 2^8 beyond which the accumulated output is
    rescaled: for every row, for one row in five (the others of its warp stay); and for none (large keys first).
    (The largest of 64 unit normals is about 2.4, 3.5 in log2 units: a growth of 4 raises it by about 14 from one 64 keys to the next, a
    growth of 2 only by 7, and then no more than a tenth of the causal rows move three times with key blocks of 64. For none: that
    maximum is hardly ever below 1 and the largest of all products below 6, so keys nine times as large stay ahead.)"""
    hq, hkv = 4, 2
    at = torch.arange(Sk, device="cuda")
    grow = torch.where(at < 64, 9.0, 1.0) if rows == "none" else 1.0 + 4.0 * (at // 64)
    q, k, v = rnd(2, Sq, hq, d, seed=1), rnd(2, Sk, hkv, d, seed=2), rnd(2, Sk, hkv, d, seed=3)
    k = (k.float() * grow[:, None, None]).to(torch.bfloat16)
    large = torch.arange(Sq, device="cuda") % (5 if rows == "some" else 1) == 0
    q = (q.float() * large[:, None, None]).to(torch.bfloat16)
    scale = 1.0 / math.sqrt(d)
    s = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float().repeat_interleave(hq // hkv, 2)) * scale * math.log2(math.e)
    if causal:
        s = s.masked_fill(torch.ones(Sq, Sk, device="cuda", dtype=torch.bool).triu(1), -math.inf)
    blocks = torch.stack([b.amax(-1) for b in s.split(128 if d == 64 else 64, dim=-1)])
    moves = (blocks[1:] > blocks.cummax(0).values[:-1] + 8).sum(0)
    often = (moves >= (2 if d == 64 else 3)).float().mean(dim=(0, 1))          # share of the batch and heads, per row
    assert moves.max() == 0 if rows == "none" else (often[large].mean() > 0.25 and not often[~large].any()), "the inputs miss their purpose"
    o, lse = C.attention_fwd(q, k, v, causal, scale)
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    o_ref, lse_ref = ref.attention_fwd(q, k, v, causal, scale)
    # scores up to a few hundred with fp32 sums (2^-24 of the sum of their terms' sizes); probabilities rounded to bf16 (2^-9)
    torch.testing.assert_close(lse, lse_ref, rtol=1e-5, atol=1e-3)
    torch.testing.assert_close(o.float(), o_ref.float(), rtol=2e-2, atol=2e-2)


def test_attention_forward_row_sums_keep_their_order(C):
    """One probability of 1 and 64 that vanish beside it when they are added one by one: a row's sum is that of its neighbour pairs
    in four running sums (every fourth pair), so exactly the sixteen of the first running sum get lost."""
    d, keys = 64, 128
    q, k = torch.zeros(1, 130, 1, d), torch.zeros(1, keys, 1, d)
    q[..., 0] = 1.0
    k[0, :, 0, 0] = torch.where(torch.arange(keys) % 2 == 1, -24.125, -300.0)
    k[0, 0, 0, 0] = 0.0
    q, k = q.to(torch.bfloat16).cuda(), k.to(torch.bfloat16).cuda()
    _, lse = C.attention_fwd(q, k, torch.randn_like(k), False, math.log(2.0))
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    p = torch.exp2(k[0, :, 0, 0].float().cpu())
    pairs, run = p[0::2] + p[1::2], torch.zeros(4)
    for i in range(0, keys // 2, 4):
        run = run + pairs[i:i + 4]
    want = torch.log(((run[0] + run[1]) + (run[2] + run[3])).double())
    # the logarithm's error is at most 2^-21.4 = 3.6e-7 there; a sum that keeps the sixteen is off by 16 * 2^-24.125 = 8.7e-7
    torch.testing.assert_close(lse.double().cpu(), want.expand(lse.shape), rtol=0, atol=4e-7)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("Sq,Sk,group,causal", [(1, 1, 1, True), (127, 127, 3, True), (129, 129, 1, True), (385, 385, 4, True),
                                                (640, 640, 2, True), (128, 300, 1, True), (65, 257, 3, False), (513, 64, 2, False)])
def test_attention_backward_at_tile_and_ring_edges(C, Sq, Sk, group, causal, d):
    """One step, a step more or less than the operand rings hold, ragged last blocks on either side, keys no query sees."""
    q, k, v = rnd(2, Sq, 2 * group, d, seed=1), rnd(2, Sk, 2, d, seed=2), rnd(2, Sk, 2, d, seed=3)
    do = rnd(2, Sq, 2 * group, d, seed=4)
    scale = 1.0 / math.sqrt(d)
    o_ref, lse_ref = ref.attention_fwd(q, k, v, causal, scale)
    want = ref.attention_bwd(do, q, k, v, o_ref, lse_ref, causal, scale)
    got = C.attention_bwd(do, q, k, v, o_ref, lse_ref, causal, scale)
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    # P and dS are rounded to bf16 (2^-9) before the second matrix products: the error of a sum of such terms stays below
    # 2^-9 of the root of its sum of squares, with a factor of four for the cancellation in dS
    for name, g, w in zip(("dq", "dk", "dv"), got, want):
        err = float((g.float() - w).norm())
        assert err <= 1e-2 * float(w.norm()) + 2e-3 * w.numel() ** 0.5, f"{name}: {err} of {float(w.norm())}"


@pytest.mark.parametrize("d,Sq,Sk,group,causal", [(64, 300, 300, 3, True), (64, 130, 400, 4, True), (64, 257, 129, 6, False), (64, 700, 700, 8, True),
                                                  (128, 520, 520, 2, True), (128, 260, 300, 4, False), (64, 300, 300, 5, True)])
@pytest.mark.parametrize("rope", [False, True])
def test_attention_backward_of_few_key_blocks_with_long_groups(C, d, Sq, Sk, group, causal, rope):
    """Key blocks whose query heads are shared by the CTAs of a cluster (groups of 3, 4, 6, 8 and 2), one whose group cannot be cut (5), and keys no
    query sees; dK and dV repeat to the bit (their sums have an order)."""
    if rope and Sq != Sk:
        pytest.skip("the fused rotation is that of self-attention")
    q, k, v = rnd(2, Sq, 2 * group, d, seed=1), rnd(2, Sk, 2, d, seed=2), rnd(2, Sk, 2, d, seed=3)
    do = rnd(2, Sq, 2 * group, d, seed=4)
    scale = 1.0 / math.sqrt(d)
    o_ref, lse_ref = ref.attention_fwd(q, k, v, causal, scale)
    want = list(ref.attention_bwd(do, q, k, v, o_ref, lse_ref, causal, scale))
    tables = ref.rope_tables(Sk, d, 10000.0, device="cuda") if rope else (None, None)
    if rope:
        for i, h in ((0, 2 * group), (1, 2)):
            want[i] = ref.rope_(want[i].reshape(2 * Sk, h * d).clone(), *tables, h, d, Sk, True).view(2, Sk, h, d)
    got = C.attention_bwd(do, q, k, v, o_ref, lse_ref, causal, scale, None, None, *tables)
    again = C.attention_bwd(do, q, k, v, o_ref, lse_ref, causal, scale, None, None, *tables)
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    assert torch.equal(got[1], again[1]) and torch.equal(got[2], again[2])
    for name, g, w in zip(("dq", "dk", "dv"), got, want):          # (bounds as above)
        err = float((g.float() - w.float()).norm())
        assert err <= 1e-2 * float(w.float().norm()) + 2e-3 * w.numel() ** 0.5, f"{name}: {err} of {float(w.float().norm())}"


# us by CTAs that share a key block's query heads, on a device with 148 SMs that says it holds 74 clusters of two or 45 of three
MEASURED_PARTS = [
    # B, S, query heads, key/value heads, d, causal
    (3, 601, 9, 3, 64, True, {1: 34.5, 3: 28.7}),
    (3, 601, 9, 3, 64, False, {1: 34.8, 3: 38.1}),           # 45 blocks of one length: two waves
    (8, 256, 9, 3, 64, True, {1: 21.0, 3: 29.1}),
    (8, 200, 9, 3, 64, False, {1: 20.2, 3: 30.5}),
    (3, 384, 15, 5, 64, True, {1: 25.6, 3: 28.7}),
    (3, 384, 15, 5, 64, False, {1: 25.8, 3: 33.3}),
    (4, 256, 9, 3, 64, False, {1: 18.7, 3: 19.9}),
    (8, 64, 6, 1, 64, True, {1: 16.9, 2: 16.4, 3: 15.6}),
    (8, 384, 12, 2, 64, True, {1: 40.4, 2: 32.3, 3: 34.6}),
    (3, 1024, 12, 2, 64, True, {1: 85.5, 2: 55.8, 3: 44.0}),
    (3, 1024, 12, 2, 64, False, {1: 88.3, 2: 57.3, 3: 76.5}),
    (4, 256, 32, 8, 64, True, {1: 25.1, 2: 24.1}),
    (8, 128, 32, 8, 64, True, {1: 19.2, 2: 20.7}),
    (1, 1024, 32, 8, 128, False, {1: 92.2, 2: 61.9}),
    (2, 601, 32, 8, 128, False, {1: 64.9, 2: 81.7}),
]


@pytest.mark.parametrize("B,S,hq,hkv,d,causal,us", MEASURED_PARTS)
def test_attention_backward_shares_key_blocks_where_it_is_faster(C, B, S, hq, hkv, d, causal, us):
    parts = C.attention_bwd_parts(B, S, S, hq, hkv, d, causal, 1, 148, 74, 45)
    assert parts in us and us[parts] <= 1.03 * min(us.values()), parts
    assert C.attention_bwd_parts(B, S, S, hq, hkv, d, causal, 1, 148, 0, 0) == 1          # a device that holds no clusters
    assert C.attention_bwd_parts(B, S, S, hq, hkv, d, causal, 1, 148, 74, 0) < 3


@pytest.mark.parametrize("largest", [3, 1])
@pytest.mark.parametrize("d,group,S,n,causal", [(64, 6, 300, 3, True), (64, 4, 260, 2, False), (128, 4, 200, 3, True), (128, 2, 520, 1, True)])
def test_attention_of_several_key_segments_with_long_groups(C, d, group, S, n, causal, largest):
    """Context parallelism's shape on local memory: keys and values in segments (the causal mask runs through the last one), fp32 dK and dV
    per segment; the query heads of a key block are shared by the CTAs of a cluster, or not."""
    B, hkv = 1, 2
    hq, scale = hkv * group, 1.0 / math.sqrt(d)
    q, do = rnd(B, S, hq, d, seed=1), rnd(B, S, hq, d, seed=2)
    ks, vs = [rnd(B, S, hkv, d, seed=3 + i) for i in range(n)], [rnd(B, S, hkv, d, seed=30 + i) for i in range(n)]
    Q, K, V = (t.float().transpose(1, 2).requires_grad_() for t in (q, torch.cat(ks, 1), torch.cat(vs, 1)))
    s = Q @ K.repeat_interleave(group, 1).transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(S, n * S, device="cuda", dtype=torch.bool).triu((n - 1) * S + 1), -math.inf)
    o_ref = s.softmax(-1) @ V.repeat_interleave(group, 1)
    o_ref.backward(do.float().transpose(1, 2))
    kp, vp = [t.data_ptr() for t in ks], [t.data_ptr() for t in vs]
    per = B * S * hkv * d
    part = torch.full((n, 2, B, S, hkv, d), float("nan"), device="cuda")
    try:
        C.attention_set_clusters(largest)
        o, lse = C.attention_fwd_segs(q, kp, vp, S, hkv, hkv * d, causal, scale)
        dq = C.attention_bwd_segs(do, q, kp, vp, S, hkv, hkv * d, o, lse, None, part.data_ptr(), 2 * per, causal, scale)
    finally:
        C.attention_set_clusters(3)
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    torch.testing.assert_close(o.float(), o_ref.transpose(1, 2), rtol=2e-2, atol=2e-2)
    back = lambda t: t.transpose(1, 2)                              # noqa: E731
    dk, dv = torch.cat(list(part[:, 0]), 1), torch.cat(list(part[:, 1]), 1)
    for name, g, w in (("dq", dq, back(Q.grad)), ("dk", dk, back(K.grad)), ("dv", dv, back(V.grad))):          # (bounds as above)
        err = float((g.float() - w).norm())
        assert err <= 1e-2 * float(w.norm()) + 2e-3 * w.numel() ** 0.5, f"{name}: {err} of {float(w.norm())}"


@pytest.mark.parametrize("d,group", [(64, 6), (128, 4)])
@pytest.mark.parametrize("largest", [1, 2])
def test_attention_backward_where_large_clusters_cannot_be_had(C, d, group, largest):
    """Key blocks whose query heads two or three CTAs would share, on a device that places smaller clusters only, or none: the next smaller number
    of CTAs, which gives the same gradients."""
    q, k, v, do = rnd(1, 400, 2 * group, d, seed=1), rnd(1, 400, 2, d, seed=2), rnd(1, 400, 2, d, seed=3), rnd(1, 400, 2 * group, d, seed=4)
    scale = 1.0 / math.sqrt(d)
    o_ref, lse_ref = ref.attention_fwd(q, k, v, True, scale)
    want = ref.attention_bwd(do, q, k, v, o_ref, lse_ref, True, scale)
    try:
        C.attention_set_clusters(largest)
        got = C.attention_bwd(do, q, k, v, o_ref, lse_ref, True, scale)
    finally:
        C.attention_set_clusters(3)
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    for name, g, w in zip(("dq", "dk", "dv"), got, want):          # (bounds as above)
        err = float((g.float() - w.float()).norm())
        assert err <= 1e-2 * float(w.float().norm()) + 2e-3 * w.numel() ** 0.5, f"{name}: {err} of {float(w.float().norm())}"


@pytest.mark.parametrize("B,S,hq,hkv,d", [(2, 256, 4, 2, 64), (1, 300, 4, 4, 64), (2, 256, 2, 1, 128), (3, 128, 2, 2, 64)])
def test_attention_backward_with_inverse_rope_on_dq_dk(C, B, S, hq, hkv, d):
    """dq / dk un-rotated inside the backward (dq in the fp32->bf16 conversion, dk in the epilogue) vs the RoPE kernel."""
    q, k, v = rnd(B, S, hq, d, seed=1), rnd(B, S, hkv, d, seed=2), rnd(B, S, hkv, d, seed=3)
    do = rnd(B, S, hq, d, seed=4)
    scale = 1.0 / math.sqrt(d)
    o_ref, lse_ref = ref.attention_fwd(q, k, v, True, scale)
    dq_r, dk_r, dv_r = ref.attention_bwd(do, q, k, v, o_ref, lse_ref, True, scale)
    cos, sin = ref.rope_tables(S + 40, d, 10000.0, device="cuda")        # a table longer than the sequence
    want_q = ref.rope_(dq_r.reshape(B * S, hq * d).clone(), cos, sin, hq, d, S, True).view(B, S, hq, d)
    want_k = ref.rope_(dk_r.reshape(B * S, hkv * d).clone(), cos, sin, hkv, d, S, True).view(B, S, hkv, d)
    dq, dk, dv = C.attention_bwd(do, q, k, v, o_ref, lse_ref, True, scale, None, None, cos, sin)
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    for name, got, want in (("dq", dq, want_q), ("dk", dk, want_k), ("dv", dv, dv_r)):
        err = float((got.float() - want.float()).norm() / (want.float().norm() + 1e-12))
        assert err < 2e-2, f"{name}: relative error {err:.4f}"


def test_phase_profiling_variant_gives_the_same_results_and_counts_cycles(C):
    B, S, hq, hkv, d = 2, 512, 4, 2, 64
    q, k, v, do = rnd(B, S, hq, d, seed=1), rnd(B, S, hkv, d, seed=2), rnd(B, S, hkv, d, seed=3), rnd(B, S, hq, d, seed=4)
    scale = 1.0 / math.sqrt(d)
    o, lse = C.attention_fwd(q, k, v, True, scale)
    dq, dk, dv = C.attention_bwd(do, q, k, v, o, lse, True, scale)
    counters = torch.zeros(16, dtype=torch.int64, device="cuda")
    C.attention_set_profile(counters)
    try:
        o2, lse2 = C.attention_fwd(q, k, v, True, scale)
        dq2, dk2, dv2 = C.attention_bwd(do, q, k, v, o, lse, True, scale)
        torch.cuda.synchronize()
    finally:
        C.attention_set_profile(None)
    assert C.kernel_status() == 0
    # a separately compiled instantiation: same algorithm, fp32 sums may be associated differently by a few ulp
    torch.testing.assert_close(o2.float(), o.float(), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(lse2, lse, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(dk2.float(), dk.float(), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(dv2.float(), dv.float(), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(dq2.float(), dq.float(), rtol=1e-2, atol=1e-2)
    c = counters.tolist()
    ctas_fwd, ctas_bwd = B * hq * (S // 128), B * hkv * (S // 128)
    assert c[13] == ctas_fwd and c[6] == ctas_bwd
    assert c[11] == B * hq * sum(range(1, S // 128 + 1))                              # causal: 1 + 2 + ... key blocks
    assert min(c[8], c[10], c[1], c[3]) > 0
    before = counters.clone()
    C.attention_fwd(q, k, v, True, scale)                                             # switched off: nothing is added
    torch.cuda.synchronize()
    assert torch.equal(counters, before)


def test_attention_on_packed_qkv_views_with_outs_and_delta(C):
    B, S, hq, hkv, d = 2, 256, 4, 2, 64
    T = B * S
    qkv = rnd(T, (hq + 2 * hkv) * d, seed=5)
    q = qkv[:, : hq * d].view(B, S, hq, d)
    k = qkv[:, hq * d:(hq + hkv) * d].view(B, S, hkv, d)
    v = qkv[:, (hq + hkv) * d:].view(B, S, hkv, d)
    scale = 1.0 / math.sqrt(d)
    o, lse = C.attention_fwd(q, k, v, True, scale)
    o_ref, lse_ref = ref.attention_fwd(q, k, v, True, scale)
    torch.testing.assert_close(o.float(), o_ref.float(), rtol=2e-2, atol=2e-2)
    do = rnd(B, S, hq, d, seed=6)
    dqkv = torch.zeros_like(qkv)
    dq = dqkv[:, : hq * d].view(B, S, hq, d)
    dk = dqkv[:, hq * d:(hq + hkv) * d].view(B, S, hkv, d)
    dv = dqkv[:, (hq + hkv) * d:].view(B, S, hkv, d)
    delta = (do.float() * o.float()).sum(-1).permute(0, 2, 1).contiguous()
    C.attention_bwd(do, q, k, v, o, lse, True, scale, delta, [dq, dk, dv])
    torch.cuda.synchronize()
    assert C.kernel_status() == 0
    dq_r, dk_r, dv_r = ref.attention_bwd(do, q, k, v, o_ref, lse_ref, True, scale)
    for got, want in ((dq, dq_r), (dk, dk_r), (dv, dv_r)):
        assert float((got.float() - want).norm() / want.norm()) < 2e-2
