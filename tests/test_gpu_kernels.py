"""sm_100a kernels against the plain-PyTorch fp32 restatements of the same ops."""
import math

import pytest
import torch

from picotron_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["pair", "pair_direct_store", "single"])
def C(request):
    """The extension with GEMMs on CTA pairs (cta_group::2; TMA-store epilogue, then per-thread stores) and on single CTAs."""
    from picotron_b200.ops import _ext
    ext = _ext.load()
    ext.set_gemm_pair(request.param != "single")
    ext.set_gemm_tma_epilogue(request.param == "pair")
    yield ext
    ext.set_gemm_pair(True)
    ext.set_gemm_tma_epilogue(True)


def _status_ok(C):
    torch.cuda.synchronize()
    assert C.kernel_status() == 0


def bf(*shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


def _rel(got, want):
    """Relative Frobenius error. bf16 inputs and one bf16 rounding of the output give ~2e-3; a dropped k-block of a small-K
    GEMM, which the element-wise tolerance below lets pass, gives 1/sqrt(number of k-blocks) or more."""
    return float((got.float() - want).norm() / (want.norm() + 1e-20))


GEMM_SHAPES = [(128, 256, 64), (128, 256, 256), (256, 512, 320), (200, 328, 136), (64, 64, 64), (1024, 2048, 512),
               (384, 1536, 2048), (1000, 1096, 1000), (2048, 2560, 1024)]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_gemm_forward_layout(C, M, N, K):
    x, w = bf(M, K, seed=1), bf(N, K, seed=2)
    y = C.gemm(x, w, False, False)
    _status_ok(C)
    want = x.float() @ w.float().t()
    torch.testing.assert_close(y.float(), want, rtol=2e-2, atol=2e-2 * math.sqrt(K))
    assert _rel(y, want) < 4e-3


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_gemm_dgrad_layout(C, M, N, K):
    dy, w = bf(M, K, seed=3), bf(K, N, seed=4)          # D[M,N] = dy[M,K] @ w[K,N]
    y = C.gemm(dy, w, False, True)
    _status_ok(C)
    want = dy.float() @ w.float()
    torch.testing.assert_close(y.float(), want, rtol=2e-2, atol=2e-2 * math.sqrt(K))
    assert _rel(y, want) < 4e-3


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_gemm_wgrad_layout_and_fp32_accumulate(C, M, N, K):
    a, b = bf(K, M, seed=5), bf(K, N, seed=6)            # D[M,N] = a^T b
    want = a.float().t() @ b.float()
    y = C.gemm(a, b, True, True)
    _status_ok(C)
    torch.testing.assert_close(y.float(), want, rtol=2e-2, atol=2e-2 * math.sqrt(K))
    assert _rel(y, want) < 4e-3
    acc = torch.full((M, N), 0.5, device="cuda", dtype=torch.float32)
    C.gemm(a, b, True, True, acc, True)
    C.gemm(a, b, True, True, acc, True)
    _status_ok(C)
    torch.testing.assert_close(acc, 0.5 + 2 * want, rtol=1e-3, atol=1e-3 * math.sqrt(K))
    assert _rel(acc - 0.5, 2 * want) < 1e-4                   # fp32 accumulation: only the bf16 inputs round


@pytest.mark.parametrize("M,N,K", [(256, 256, 512), (256, 256, 511), (264, 520, 449), (576, 576, 8192), (8, 8, 16384), (1024, 512, 577)])
def test_gemm_fp32_accumulation_with_k_split_over_cta_pairs(M, N, K):
    """Few output tiles and a long reduction: several CTA pairs add their part of K to one tile (remainders of the split,
    a last k-block of one row, tiles that stick out of the matrix)."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    a, b = bf(K, M, seed=71), bf(K, N, seed=72)
    acc = torch.full((M, N), 0.5, device="cuda", dtype=torch.float32)
    C.gemm(a, b, True, True, acc, True)
    _status_ok(C)
    # fp32 sums of K products in another order: error of order sqrt(K) * 2^-24 of the sum's size sqrt(K)
    assert _rel(acc - 0.5, a.double().t() @ b.double()) < 1e-5


@pytest.mark.parametrize("M,N,K", [(576, 576, 8192), (573, 569, 4100), (264, 520, 32768), (8, 8, 16384)])
def test_gemm_weight_gradient_parts_are_repeatable_and_rounded_once(C, M, N, K):
    """The parts of K add up in a fixed order and reach the destination in one addition, also where rows and columns end within a
    tile, a quad of columns and a strided destination."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    wide = lambda n: (n + 7) // 8 * 8
    a, b = bf(K, wide(M), seed=81)[:, :M], bf(K, wide(N), seed=82)[:, :N]
    want = a.double().t() @ b.double()
    base = 2.0 ** 20
    first = None
    for _ in range(12):
        big = torch.full((M, wide(N) + 8), base, device="cuda")
        n0 = C.launch_count()
        C.gemm(a, b, True, True, big[:, :N], True)
        assert C.launch_count() - n0 == 2, "this shape should be split"
        first = big if first is None else first
        assert torch.equal(big, first)
    _status_ok(C)
    assert bool((big[:, N:] == base).all())
    # one rounding at 2^20 (half an ulp: 2^-4) of a sum that is itself good to 1e-5 of its size
    err = float((big[:, :N].double() - base - want).abs().max())
    assert err <= 2 ** -4 + 1e-5 * float(want.abs().max()), err


@pytest.mark.parametrize("tile_n", [128, 192, 256])
@pytest.mark.parametrize("parts", [1, 2, 7])
@pytest.mark.parametrize("M,N,K", [(8, 8, 1024), (264, 520, 448), (600, 584, 1000), (256, 128, 512), (1000, 72, 640), (304, 576, 192)])
def test_gemm_tile_widths_and_parts_of_every_layout(tile_n, parts, M, N, K):
    """Every tile width, unsplit and with K in parts (uneven ones, a last k-block of 8 to 40 rows, tiles beyond the matrix), for the
    forward layout with and without a residual, input gradients and fp32 accumulation."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    x, w, wt, res, xt = bf(M, K, seed=1), bf(N, K, seed=2), bf(K, N, seed=3), bf(M, N, seed=4), bf(K, M, seed=5)
    acc = torch.full((M, N), 0.5, device="cuda")
    try:
        C.set_gemm_tile_n(tile_n)
        if parts > 1:
            C.set_gemm_split_parts(parts)
        else:
            C.set_gemm_split_dgrad(False)
        C.gemm(xt, wt, True, True, acc, True)
        got = [C.gemm(x, w, False, False), C.gemm_add(x, w, res), C.gemm(x, wt, False, True)]
        if N % 64 == 0:                                       # the SwiGLU backward is never split: equal, whatever the width
            gu = bf(M, 2 * N, seed=6)
            dgu = C.gemm_dgrad_swiglu_bwd(x, wt, gu)
            C.set_gemm_tile_n(256)
            assert torch.equal(dgu, C.gemm_dgrad_swiglu_bwd(x, wt, gu))
    finally:
        C.set_gemm_tile_n(0)
        C.set_gemm_split_parts(0)
    _status_ok(C)
    y = x.double() @ w.double().t()
    for g, want in zip(got, [y, y + res.double(), x.double() @ wt.double()]):
        assert _rel(g.double(), want) < 4e-3                  # one bf16 rounding of the result
    # fp32 sums in another order (sqrt(K) * 2^-24 of their size) and 0.5 added to them
    assert _rel(acc.double() - 0.5, xt.double().t() @ wt.double()) < 1e-5


@pytest.mark.parametrize("M,N,K", [(8, 8, 72), (264, 520, 448), (600, 584, 1000), (256, 64, 512), (1000, 136, 640), (225, 200, 1480), (512, 2048, 8192)])
def test_gemm_with_k_shared_in_clusters(C, M, N, K):
    """Two CTA pairs per tile, each half of K: tiles beyond the matrix, second halves of a tile with no column or eight, an odd number of
    k-blocks, a last one of 8 rows; output and residual are rows of wider tensors, whose other columns stay as they were."""
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    x, w, wt, wide = bf(M, K, seed=1), bf(N, K, seed=2), bf(K, N, seed=3), bf(M, N + 16, seed=4)
    res = wide[:, 8:8 + N]
    runs = []
    try:
        C.set_gemm_cluster(2)
        for _ in range(3):
            big = torch.full((M, N + 16), 3.0, device="cuda", dtype=torch.bfloat16)
            n0 = C.launch_count()
            C.gemm(x, wt, False, True, big[:, 8:8 + N], False)
            runs.append([C.gemm(x, w, False, False), C.gemm_add(x, w, res), big])
            assert C.launch_count() - n0 == 3
        C.set_gemm_cluster(1)
        C.set_gemm_split_dgrad(False)
        whole = [C.gemm(x, w, False, False), C.gemm_add(x, w, res), C.gemm(x, wt, False, True)]
    finally:
        C.set_gemm_cluster(0)
        C.set_gemm_split_dgrad(True)
    _status_ok(C)
    for run in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(run, runs[0]))
    got = runs[0][:2] + [runs[0][2][:, 8:8 + N]]
    assert bool((runs[0][2][:, :8] == 3).all()) and bool((runs[0][2][:, 8 + N:] == 3).all())
    y = x.double() @ w.double().t()
    for g, one, want in zip(got, whole, [y, y + res.double(), x.double() @ wt.double()]):
        # one bf16 rounding of the result (2^-9 of each value at most); the sums' order changes it for those at the edge of a rounding only
        assert _rel(g.double(), want) < 2.5e-3 and _rel(g.double(), want) < 1.01 * _rel(one.double(), want) + 1e-5


@pytest.mark.parametrize("kind,M,N,K,shared", [("fwd", 256, 576, 1536, True), ("add", 256, 960, 1024, True), ("dgrad", 384, 2048, 6144, True),
                                               ("fwd", 512, 2048, 8192, True), ("dgrad", 256, 2048, 3072, True), ("fwd", 256, 576, 1472, False),
                                               ("add", 256, 960, 832, False), ("dgrad", 256, 576, 1472, False), ("dgrad", 512, 2048, 8256, False),
                                               ("fwd", 1024, 2048, 2048, False), ("add", 4096, 2048, 8192, False)])
def test_gemm_shares_k_in_clusters_by_rule(kind, M, N, K, shared):
    """Shapes on both sides of the rule: few tiles and a long K share it, a short one, more tiles than clusters, and an input gradient over more
    than 8192 do not; what runs by the rule is what runs when the switch says so, and its plan tells."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the rule counts SMs")
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    x, w, wt, res = bf(M, K, seed=1), bf(N, K, seed=2), bf(K, N, seed=3), bf(M, N, seed=4)
    call = {"fwd": lambda: C.gemm(x, w, False, False), "add": lambda: C.gemm_add(x, w, res), "dgrad": lambda: C.gemm(x, wt, False, True)}[kind]
    assert (C.gemm_plan(kind, M, N, K) == (128, -2)) == shared
    by_rule = call()
    try:
        C.set_gemm_cluster(2 if shared else 1)
        assert torch.equal(by_rule, call())
        C.set_gemm_cluster(1 if shared else 2)
        assert not torch.equal(by_rule, call())               # (the other order of the sums moves a few roundings)
    finally:
        C.set_gemm_cluster(0)
    _status_ok(C)


def test_gemm_over_nothing_is_zero(C):
    """The weight gradient of an empty batch: zeros, or what the destination holds where it is added to."""
    dy, x = bf(0, 72), bf(0, 136)
    stale = [torch.full((72, 136), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(4)]
    del stale                                                 # (the allocator hands the same memory out again)
    assert torch.count_nonzero(C.gemm(dy, x, True, True)) == 0
    acc = torch.full((72, 136), 0.5, device="cuda")
    assert C.gemm(dy, x, True, True, acc, True).eq(0.5).all()
    assert C.gemm(dy, x, True, True, acc, False).eq(0.0).all()
    assert C.gemm(x, bf(200, 136), False, False).shape == (0, 200)


# us by (columns of a tile, parts; -2: shared within clusters), operands not in L2
MEASURED_PLANS = [
    ("swiglu_bwd", 1024, 11008, 4096, {(128, 1): 101.0, (192, 1): 98.2, (256, 1): 86.1}),
    ("swiglu_bwd", 768, 14336, 4096, {(128, 1): 102.4, (256, 1): 88.1}),
    ("swiglu_bwd", 2048, 8192, 2048, {(128, 1): 81.9, (192, 1): 73.7, (256, 1): 69.7}),
    ("swiglu", 512, 22016, 4096, {(128, 1): 92.6, (256, 1): 81.9}),
    ("rope", 512, 12288, 4096, {(128, 1): 59.5, (256, 1): 55.3}),
    ("dgrad", 1024, 2048, 16384, {(128, 1): 65.8, (256, 2): 60.4}),
    ("dgrad", 512, 4096, 12288, {(128, 1): 57.3, (256, 2): 52.9}),
    ("wgrad", 2048, 512, 8192, {(128, 2): 29.6, (256, 4): 27.6, (192, 3): 27.6}),
    ("fwd", 128, 4096, 4096, {(128, -2): 18.8, (128, 2): 21.5, (128, 1): 22.9}),
    ("add", 512, 2048, 8192, {(128, -2): 26.7, (256, 4): 29.7, (128, 1): 34.9}),
    ("dgrad", 384, 2048, 6144, {(128, -2): 20.8, (256, 4): 25.6, (128, 2): 24.7}),
    ("dgrad", 4096, 576, 3072, {(256, 1): 20.7, (128, 1): 19.8, (192, 1): 17.2}),
    ("wgrad", 49152, 576, 2048, {(256, 1): 110.0, (128, 1): 118.0, (192, 1): 102.0}),
    ("fwd", 256, 576, 576, {(256, 1): 7.1, (128, 1): 5.3}),
]


@pytest.mark.parametrize("kind,M,N,K,us", MEASURED_PLANS)
def test_gemm_tiles_and_parts_are_the_fastest_measured(kind, M, N, K, us):
    """The rule's choice among plans that were measured (3 %: what runs of one plan differ by)."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("measured on 148 SMs")
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    plan = tuple(C.gemm_plan(kind, M, N, K))
    assert plan in us and us[plan] <= 1.03 * min(us.values()), plan


@pytest.mark.parametrize("T,N,K", [(64, 576, 49152), (500, 520, 16392), (300, 2048, 16384)])
def test_gemm_input_gradient_parts_are_repeatable(C, T, N, K):
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    dy, w = bf(T, K, seed=1, scale=0.1), bf(K, N, seed=2, scale=0.1)
    first = C.gemm(dy, w, False, True)
    for _ in range(12):
        assert torch.equal(C.gemm(dy, w, False, True), first)
    _status_ok(C)


@pytest.mark.parametrize("T,I,K", [(256, 128, 64), (300, 384, 320), (1024, 2048, 512), (4096, 1024, 2048)])
def test_gemm_with_swiglu_epilogue(T, I, K):
    """gate/up GEMM whose epilogue also writes silu(gate) * up, against the two separate kernels and fp32 math."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    x, w = bf(T, K, seed=21), bf(2 * I, K, seed=22, scale=0.5)
    r = C.gemm_swiglu(x, w)
    assert r, "the fused kernel should cover this shape"
    gu, h = r
    _status_ok(C)
    gu_ref = C.gemm(x, w, False, False)
    torch.testing.assert_close(gu.float(), gu_ref.float(), rtol=0, atol=0)            # same accumulators, same rounding
    torch.testing.assert_close(gu.float(), x.float() @ w.float().t(), rtol=2e-2, atol=2e-2 * math.sqrt(K))
    torch.testing.assert_close(h.float(), ref.swiglu_fwd(gu).float(), rtol=2e-2, atol=2e-2)
    assert C.gemm_swiglu(x, bf(2 * 72, K, seed=23)) == []                             # I % 128 != 0: not covered


@pytest.mark.parametrize("T,V,K,vocab_start", [(256, 512, 64, 0), (300, 1000, 192, 0), (2048, 49152, 2048, 0), (512, 4096, 256, 4096),
                                               (32, 48, 256, 0), (200, 1000, 64, 1000)])
def test_lm_head_gemm_with_cross_entropy_statistics_epilogue(T, V, K, vocab_start):
    """Logits GEMM whose epilogue produces row max / sum-exp / target logit, against the separate statistics kernel (which
    reads the same stored logits) and against fp32 math."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    x, w = bf(T, K, seed=61), bf(V, K, seed=62, scale=0.3)
    g = torch.Generator(device="cuda").manual_seed(63)
    targets = torch.randint(0, 2 * V if vocab_start else V, (T,), device="cuda", generator=g)   # some outside this shard
    r = C.gemm_ce_stats(x, w, targets, vocab_start)
    assert r, "the fused kernel should cover this shape"
    logits, rowmax, sumexp, tgt = r
    _status_ok(C)
    plain = C.gemm(x, w, False, False)
    torch.testing.assert_close(logits.float(), plain.float(), rtol=0, atol=0)
    m2, s2, t2 = C.ce_stats(plain, targets, vocab_start)
    torch.testing.assert_close(rowmax, m2, rtol=0, atol=0)
    torch.testing.assert_close(sumexp, s2, rtol=2e-3, atol=1e-3)
    torch.testing.assert_close(tgt, t2, rtol=0, atol=0)
    lse_ref = torch.logsumexp(x.float() @ w.float().t(), dim=-1)
    torch.testing.assert_close(rowmax + torch.log(sumexp), lse_ref, rtol=1e-2, atol=3e-2)


@pytest.mark.parametrize("T,V,K,vocab_start", [(1, 8, 64, 0), (300, 1000, 192, 0), (257, 8456, 128, 0), (200, 1000, 64, 1000), (64, 128256, 64, 0)])
def test_lm_head_loss_from_two_kernels(T, V, K, vocab_start):
    """Loss terms and in-place gradient straight from the GEMM's tile statistics (one tile, a partial last one, more tiles than lanes;
    targets outside the shard count as logit 0), with and without the gradient, against 64-bit arithmetic on the stored logits."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    x, w = bf(T, K, seed=91), bf(V, K, seed=92, scale=0.3)
    g = torch.Generator(device="cuda").manual_seed(93)
    targets = torch.randint(0, vocab_start + V, (T,), device="cuda", generator=g)
    logits = C.gemm(x, w, False, False).double()
    lse = torch.logsumexp(logits, -1)
    col = targets - vocab_start
    inside = (col >= 0) & (col < V)
    hot = torch.nn.functional.one_hot(col.clamp(0, V - 1), V) * inside[:, None]
    terms = [torch.full((T,), float("nan"), device="cuda") for _ in range(2)]
    got = C.gemm_ce_loss(x, w, targets, vocab_start, 0.25, terms[0], True)
    none = C.gemm_ce_loss(x, w, targets, vocab_start, 0.25, terms[1], False)
    _status_ok(C)
    assert none.numel() == 0 and torch.equal(terms[0], terms[1])
    # fp32 sums of V exponentials good to 2^-22 each, and lse itself rounded to fp32: a few 1e-6 of |lse| + 1
    want = lse - (logits * hot).sum(-1)
    assert float(((terms[0].double() - want).abs() / (1 + lse.abs())).max()) < 5e-6
    want = (torch.exp(logits - lse[:, None]) - hot) * 0.25
    assert float((got.double() - want).norm() / want.norm()) < 4e-3                  # one bf16 rounding


@pytest.mark.parametrize("T,V,K,vocab_start", [(2048, 2048, 512, 0), (600, 1000, 192, 1000), (1024, 8456, 128, 0), (256, 128256, 64, 0)])
def test_lm_head_loss_is_that_of_the_separate_kernels_to_the_bit(T, V, K, vocab_start):
    """The log-sum-exp is the row maximum plus torch.log of the sum in fp32, so loss terms and gradient do not depend on whether one
    kernel finishes the statistics or several do."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    x, w = bf(T, K, seed=94), bf(V, K, seed=95, scale=0.3)
    targets = torch.randint(0, vocab_start + V, (T,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(96))
    logits, rowmax, sumexp, tgt = C.gemm_ce_stats(x, w, targets, vocab_start)
    lse = rowmax + torch.log(sumexp)
    terms = torch.empty(T, device="cuda")
    got = C.gemm_ce_loss(x, w, targets, vocab_start, 0.25, terms, True)
    C.ce_grad_(logits, targets, lse, 0.25, vocab_start)
    _status_ok(C)
    assert torch.equal(terms, lse - tgt)
    assert torch.equal(got, logits)


@pytest.mark.parametrize("T,N,K", [(256, 256, 64), (300, 328, 320), (1024, 2048, 512), (4096, 2048, 8192), (200, 72, 136)])
def test_gemm_with_residual_add_epilogue(T, N, K):
    """Projection + residual add from one GEMM (the epilogue fetches the residual tile) against GEMM followed by the add."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    x, w, res = bf(T, K, seed=41), bf(N, K, seed=42, scale=0.5), bf(T, N, seed=43, scale=4.0)
    got = C.gemm_add(x, w, res)
    assert got is not None, "the fused kernel should cover this shape"
    _status_ok(C)
    want = x.float() @ w.float().t() + res.float()
    torch.testing.assert_close(got.float(), want, rtol=2e-2, atol=2e-2 * math.sqrt(K))
    assert _rel(got, want) < 4e-3
    two_step = C.add(res, C.gemm(x, w, False, False))
    assert _rel(got, want) <= _rel(two_step, want) + 1e-4       # one rounding instead of two


@pytest.mark.parametrize("T,I,H", [(256, 256, 64), (300, 320, 192), (1024, 2048, 512), (4096, 8192, 2048), (512, 5504, 1024)])
def test_dgrad_gemm_with_swiglu_backward_epilogue(T, I, H):
    """Down-projection dgrad whose epilogue applies the SwiGLU backward, against dgrad GEMM + activation-backward kernel
    and against fp32 math."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    dy, w, gu = bf(T, H, seed=51), bf(H, I, seed=52, scale=0.5), bf(T, 2 * I, seed=53, scale=1.5)
    got = C.gemm_dgrad_swiglu_bwd(dy, w, gu)
    assert got is not None, "the fused kernel should cover this shape"
    _status_ok(C)
    da = dy.float() @ w.float()
    g, u = gu[:, :I].float(), gu[:, I:].float()
    sig = torch.sigmoid(g)
    want = torch.cat([da * u * sig * (1 + g * (1 - sig)), da * g * sig], dim=1)
    assert _rel(got, want) < 6e-3
    two_step = C.swiglu_bwd(gu, C.gemm(dy, w, False, True))
    assert _rel(got, want) <= _rel(two_step, want) + 1e-4       # da is not rounded to bf16 on the way
    torch.testing.assert_close(got.float(), two_step.float(), rtol=5e-2, atol=5e-2 * math.sqrt(H))
    assert C.gemm_dgrad_swiglu_bwd(dy, bf(H, 72, seed=54), bf(T, 144, seed=55)) is None      # I % 64 != 0: not covered


@pytest.mark.parametrize("up,da", [(64.0, 2.0 ** -7), (2.0 ** -7, 64.0), (1.0, 2.0 ** -9)])
def test_gemm_with_swiglu_backward_epilogue_of_very_negative_gates(up, da):
    """Gates whose sigmoid is next to the smallest normal number, and the same ones positive: what `up`, the gate and the gradient make of
    it is a normal number again and no zero. Rows of one 1 make the GEMM's result the weight itself."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    T, I = 256, 64
    g = torch.linspace(-87.0, 87.0, T * I, device="cuda").view(T, I).to(torch.bfloat16)
    gu = torch.cat([g, torch.full_like(g, up)], 1).contiguous()
    got = C.gemm_dgrad_swiglu_bwd(torch.eye(T, device="cuda", dtype=torch.bfloat16), torch.full((T, I), da, device="cuda", dtype=torch.bfloat16), gu)
    _status_ok(C)
    g = g.double()
    s = torch.sigmoid(g)
    want = torch.cat([da * up * s * (1 + g * (1 - s)), da * g * s], 1)
    # bf16's rounding, and that of the exponential's argument (126 at most: 2^-18 of it, times ln 2) with a few more of 2^-24; what is below
    # the smallest normal number may be zero
    assert bool(((got.double() - want).abs() <= (2.0 ** -8) * want.abs() + 2.0 ** -126).all())


@pytest.mark.parametrize("B,S,hq,hkv,d,K", [(2, 128, 4, 2, 64, 256), (1, 200, 3, 1, 64, 192), (2, 128, 4, 2, 128, 256),
                                            (4, 1024, 32, 32, 64, 512), (1, 96, 5, 5, 128, 128)])
def test_gemm_with_rope_epilogue(B, S, hq, hkv, d, K):
    """qkv GEMM whose epilogue rotates the q and k heads, against GEMM followed by the RoPE kernel / fp32 restatement."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    N = (hq + 2 * hkv) * d
    x, w = bf(B * S, K, seed=31), bf(N, K, seed=32, scale=0.5)
    cos, sin = ref.rope_tables(S, d, 10000.0, device="cuda")
    got = C.gemm_rope(x, w, cos, sin, hq + hkv, d, S)
    assert got is not None
    _status_ok(C)
    plain = C.gemm(x, w, False, False)
    want = ref.rope_((x.float() @ w.float().t()), cos, sin, hq + hkv, d, S)          # fp32 throughout
    torch.testing.assert_close(got.float(), want, rtol=2e-2, atol=2e-2 * math.sqrt(K))
    torch.testing.assert_close(got[:, (hq + hkv) * d:].float(), plain[:, (hq + hkv) * d:].float(), rtol=0, atol=0)   # v untouched
    two_step = plain.clone()
    C.rope_(two_step, cos, sin, hq + hkv, d, S, False)
    torch.testing.assert_close(got.float(), two_step.float(), rtol=2e-2, atol=0.25)   # one rounding instead of two


@pytest.mark.parametrize("group_m", [1, 3, 8, 64])
def test_gemm_tile_numbering_group_sizes(group_m):
    """Every group size of the tile numbering visits each output tile exactly once (ragged shapes included)."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    keep = C.get_gemm_group_m()
    C.set_gemm_group_m(group_m)
    try:
        for M, N, K in [(2816, 1280, 192), (1000, 1096, 320), (256, 4096, 128)]:
            x, w = bf(M, K, seed=41), bf(N, K, seed=42)
            y = C.gemm(x, w, False, False)
            _status_ok(C)
            torch.testing.assert_close(y.float(), x.float() @ w.float().t(), rtol=2e-2, atol=2e-2 * math.sqrt(K))
    finally:
        C.set_gemm_group_m(keep)


def test_gemm_strided_rows_and_out_slice(C):
    big = bf(512, 1024, seed=7)
    x = big[:, 256:512]                                    # row stride 1024, 256 columns
    w = bf(384, 256, seed=8)
    out = torch.zeros(600, 384, device="cuda", dtype=torch.bfloat16)
    C.gemm(x, w, False, False, out[40:552], False)
    _status_ok(C)
    torch.testing.assert_close(out[40:552].float(), x.float() @ w.float().t(), rtol=2e-2, atol=0.4)
    assert float(out[:40].abs().sum()) == 0 and float(out[552:].abs().sum()) == 0


@pytest.mark.parametrize("T,H", [(7, 64), (300, 2048), (129, 4096)])
def test_rmsnorm_fwd_bwd(C, T, H):
    x, d, w = bf(T, H, seed=1), bf(T, H, seed=2), (1 + 0.1 * bf(H, seed=3).float()).to(torch.bfloat16)
    y, rstd = C.rmsnorm_fwd(x, w, 1e-5)
    y_ref, rstd_ref = ref.rmsnorm_fwd(x, w, 1e-5)
    torch.testing.assert_close(y.float(), y_ref.float(), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(rstd, rstd_ref, rtol=1e-4, atol=1e-5)
    xn, y2, rstd2 = C.add_rmsnorm_fwd(x, d, w, 1e-5)
    xn_ref, y2_ref, rstd2_ref = ref.add_rmsnorm_fwd(x, d, w, 1e-5)
    torch.testing.assert_close(xn.float(), xn_ref.float(), rtol=0, atol=0)
    torch.testing.assert_close(y2.float(), y2_ref.float(), rtol=1e-2, atol=2e-2)
    dy, dres = bf(T, H, seed=4), bf(T, H, seed=5)
    dx, dw = C.rmsnorm_bwd(dy, x, w, rstd, dres)
    dx_ref, dw_ref = ref.rmsnorm_bwd(dy, x, w, rstd_ref, dres)
    torch.testing.assert_close(dx.float(), dx_ref.float(), rtol=2e-2, atol=3e-2)
    torch.testing.assert_close(dw, dw_ref, rtol=1e-3, atol=1e-2 * math.sqrt(T))
    dx0, _ = C.rmsnorm_bwd(dy, x, w, rstd, None)
    torch.testing.assert_close(dx0.float(), ref.rmsnorm_bwd(dy, x, w, rstd_ref)[0].float(), rtol=2e-2, atol=3e-2)


@pytest.mark.parametrize("T", [1, 9, 2500])
@pytest.mark.parametrize("H", [8, 256, 264, 576, 960, 1024, 1032, 1544, 2056, 3080, 4104, 8192])
def test_rmsnorm_at_the_edges_of_its_team_sizes(C, T, H):
    """Row widths on both sides of every change of threads per row and chunks per thread, with more rows than one pass covers."""
    x, d, dy = bf(T, H, seed=1), bf(T, H, seed=2), bf(T, H, seed=3)
    w = (1 + 0.1 * bf(H, seed=4).float()).to(torch.bfloat16)
    xn, y, rstd = C.add_rmsnorm_fwd(x, d, w, 1e-5)
    xn_ref, y_ref, rstd_ref = ref.add_rmsnorm_fwd(x, d, w, 1e-5)
    assert torch.equal(xn, xn_ref)
    torch.testing.assert_close(rstd, rstd_ref, rtol=1e-5, atol=0)           # fp32 sums of at most 8192 squares in another order
    torch.testing.assert_close(y, y_ref, rtol=2 ** -7, atol=0)              # bf16 neighbours
    torch.testing.assert_close(C.rmsnorm_fwd(xn, w, 1e-5)[0], y, rtol=2 ** -7, atol=0)
    acc = torch.full((H,), 0.5, device="cuda")
    dx, _ = C.rmsnorm_bwd(dy, xn, w, rstd, d, acc)
    dx_ref, dw_ref = ref.rmsnorm_bwd(dy, xn, w, rstd, d)
    # fp32 terms of size up to |dy| + |dres|, rounded once to bf16
    torch.testing.assert_close(dx.float(), dx_ref.float(), rtol=2 ** -7, atol=2e-3)
    torch.testing.assert_close(acc - 0.5, dw_ref, rtol=1e-4, atol=1e-5 * T ** 0.5 * 16)


# one width per variant of the kernel: rows a CTA works on at a time, its CTAs per SM, rows in flight per team (with_backward_team, bwd_stages)
@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("H,rows,ctas,slots", [(256, 8, 3, 4), (264, 8, 3, 2), (512, 8, 3, 2), (576, 8, 2, 2), (960, 8, 2, 2), (1032, 2, 3, 2),
                                               (2056, 1, 3, 3), (4104, 1, 2, 2)])
def test_rmsnorm_backward_with_rows_fetched_ahead(C, H, rows, ctas, slots, residual):
    """Every team goes round its ring of fetched rows more than twice, some a row further than the others."""
    teams = rows * ctas * torch.cuda.get_device_properties(0).multi_processor_count
    T = 2 * slots * teams + teams // 2 + 1
    x, dy = bf(T, H, seed=1), bf(T, H, seed=2)
    dres = bf(T, H, seed=3) if residual else None
    w = (1 + 0.1 * bf(H, seed=4).float()).to(torch.bfloat16)
    rstd = 0.5 + torch.rand(T, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    acc = torch.full((H,), 0.5, device="cuda")
    dx, _ = C.rmsnorm_bwd(dy, x, w, rstd, dres, acc)
    _status_ok(C)
    dx_ref, dw_ref = ref.rmsnorm_bwd(dy, x, w, rstd, dres)
    # fp32 terms of size up to 1.5 |dy| + |dres|, rounded once to bf16; T terms of size 1.5 |dy x| in fp32, in any order
    torch.testing.assert_close(dx.float(), dx_ref.float(), rtol=2 ** -7, atol=4e-3)
    torch.testing.assert_close(acc - 0.5, dw_ref, rtol=1e-4, atol=2e-5 * T ** 0.5 * 16)


def _row_sum_in_kernel_order(terms):
    """Sum over the last dimension of an fp32 CPU tensor in the RMSNorm kernels' order: running sums over the 8-element chunks
    c, c + 256, ..., a butterfly over 32 neighbouring ones, then the eight warp sums."""
    T, H = terms.shape
    groups = (H // 8 + 255) // 256
    c = torch.zeros(T, groups * 256 * 8)
    c[:, :H] = terms
    c = c.view(T, groups, 256, 8)
    run = torch.zeros(T, 256)
    for g in range(groups):
        for j in range(8):
            run = run + c[:, g, :, j]
    w, lanes = run.view(T, 8, 32), torch.arange(32)
    for o in (16, 8, 4, 2, 1):
        w = w + w[:, :, lanes ^ o]
    s = w[:, :, 0].unbind(1)
    return (((s[0] + s[1]) + (s[2] + s[3])) + (s[4] + s[5])) + (s[6] + s[7])


@pytest.mark.parametrize("T", [16, 1000, 2500])
@pytest.mark.parametrize("H", [576, 960, 1024, 1544, 2048, 2056, 3080, 4096, 8192])
def test_rmsnorm_row_sums_do_not_depend_on_the_threads_per_row(C, H, T):
    """Rows whose sums lose or keep whole groups of terms depending on the order of the additions; few rows get more threads each."""
    # forward: in chunks 0..31 one large square per chunk, behind which every following term of the same running sum vanishes
    x = torch.full((T, H), 0.95)
    x[:, :256:8] = 4096.0
    x = x.to(torch.bfloat16)
    one = torch.ones(H, device="cuda", dtype=torch.bfloat16)
    _, rstd = C.rmsnorm_fwd(x.cuda(), one, 1e-5)
    xn, _, rstd_add = C.add_rmsnorm_fwd(x.cuda(), torch.zeros_like(x).cuda(), one, 1e-5)
    _status_ok(C)
    want = (_row_sum_in_kernel_order(x[:1].float() ** 2).double() / H + 1e-5).rsqrt().expand(T)
    # approximate division and reciprocal root: 2 ulp of 2^-24 and 2^-22.9 relative, halved and summed; the other orders are off
    # by up to 1e-6
    for r in (rstd, rstd_add):
        torch.testing.assert_close(r.cpu().double(), want, rtol=3e-7, atol=0)
    assert torch.equal(xn.cpu(), x)
    # backward: 2^30 and -2^30 in different chunks, ones elsewhere; how many ones survive is a matter of the order
    gen = torch.Generator().manual_seed(H)
    dy = torch.ones(16, H)
    for row in dy:
        a, b = torch.randperm(H, generator=gen)[:2].tolist()
        row[a], row[b] = 2.0 ** 30, -2.0 ** 30
    want = (dy - (_row_sum_in_kernel_order(dy) / H)[:, None]).repeat(157, 1)[:T]
    dy = dy.repeat(157, 1)[:T]
    # x = w = rstd = 1: dx = dy - sum(dy) / H
    dx, _ = C.rmsnorm_bwd(dy.to(torch.bfloat16).cuda(), torch.ones(T, H, device="cuda", dtype=torch.bfloat16), one,
                          torch.ones(T, device="cuda"), None)
    _status_ok(C)
    torch.testing.assert_close(dx.float().cpu(), want, rtol=2 ** -8, atol=2 ** -8)


@pytest.mark.parametrize("T,H", [(513, 2048), (64, 768), (33, 256), (40, 4096), (9, 320)])
def test_rmsnorm_bwd_accumulates_into_fp32_destination(C, T, H):
    """dw added in place to an fp32 vector (a gradient-bucket slice), also when that slice is not 16-byte aligned."""
    x, dy, dres = bf(T, H, seed=1), bf(T, H, seed=2), bf(T, H, seed=3)
    w = (1 + 0.1 * bf(H, seed=4).float()).to(torch.bfloat16)
    _, rstd = C.rmsnorm_fwd(x, w, 1e-5)
    dx_ref, dw_ref = ref.rmsnorm_bwd(dy, x, w, rstd, dres)
    store = torch.full((H + 4,), 0.5, device="cuda", dtype=torch.float32)
    for off in (0, 1):
        acc = store[off:off + H]
        acc.fill_(0.5)
        dx, out = C.rmsnorm_bwd(dy, x, w, rstd, dres, acc)
        dx, out = C.rmsnorm_bwd(dy, x, w, rstd, dres, acc)
        _status_ok(C)
        assert out.data_ptr() == acc.data_ptr()
        torch.testing.assert_close(dx.float(), dx_ref.float(), rtol=2e-2, atol=3e-2)
        torch.testing.assert_close(acc, 0.5 + 2 * dw_ref, rtol=1e-3, atol=2e-2 * math.sqrt(T))


@pytest.mark.parametrize("d,hq,hkv", [(64, 4, 2), (128, 2, 2), (64, 32, 8), (128, 16, 5), (32, 4, 4)])
def test_rope_inplace_and_inverse(C, d, hq, hkv):
    B, S = 2, 48
    qkv = bf(B * S, (hq + 2 * hkv) * d, seed=1)
    cos, sin = ref.rope_tables(S, d, 10000.0, device="cuda")
    want = ref.rope_(qkv.clone(), cos, sin, hq + hkv, d, S)
    got = qkv.clone()
    C.rope_(got, cos, sin, hq + hkv, d, S, False)
    torch.testing.assert_close(got.float(), want.float(), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(got[:, (hq + hkv) * d:], qkv[:, (hq + hkv) * d:], rtol=0, atol=0)   # v untouched
    C.rope_(got, cos, sin, hq + hkv, d, S, True)
    torch.testing.assert_close(got.float(), qkv.float(), rtol=2e-2, atol=3e-2)


def test_swiglu(C):
    gu, da = bf(100, 2 * 512, seed=1), bf(100, 512, seed=2)
    torch.testing.assert_close(C.swiglu_fwd(gu).float(), ref.swiglu_fwd(gu).float(), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(C.swiglu_bwd(gu, da).float(), ref.swiglu_bwd(gu, da).float(), rtol=2e-2, atol=2e-2)


def test_embedding_fwd_bwd_with_vocab_shard(C):
    V, H, T = 300, 128, 500
    w = bf(V, H, seed=1)
    ids = torch.randint(0, 2 * V, (T,), device="cuda")
    out = C.embedding_fwd(ids, w, 100)
    torch.testing.assert_close(out.float(), ref.embedding_fwd(ids, w, 100).float(), rtol=0, atol=0)
    dy = bf(T, H, seed=2)
    dw = torch.zeros(V, H, device="cuda")
    C.embedding_bwd(ids, dy, dw, 100)
    want = torch.zeros(V, H, device="cuda")
    ref.embedding_bwd(ids, dy, want, 100)
    torch.testing.assert_close(dw, want, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("T,H,off", [(1, 8, 0), (37, 576, 0), (300, 2056, 0), (37, 576, 1)])
def test_embedding_backward_of_repeated_ids_and_any_alignment(C, T, H, off):
    """Rows hit by many tokens, widths that fill no block, and a gradient that does not start on 16 bytes (scalar additions)."""
    ids = torch.arange(T, device="cuda") % 5 * 7
    dy = bf(T, H, seed=3)
    dw = torch.ones(40 * H + off, device="cuda")[off:].view(40, H)
    C.embedding_bwd(ids, dy, dw, 0)
    want = torch.ones(40, H, device="cuda", dtype=torch.float64)
    want.index_add_(0, ids, dy.double())
    _status_ok(C)
    # sums of at most 60 bf16 values of size ~1 in fp32, in any order
    torch.testing.assert_close(dw.double(), want, rtol=0, atol=60 * 2.0 ** -20)


def test_embedding_backward_without_columns_does_nothing(C):
    ids = torch.zeros(5, device="cuda", dtype=torch.long)
    C.embedding_bwd(ids, torch.empty(5, 0, device="cuda", dtype=torch.bfloat16), torch.empty(3, 0, device="cuda"), 0)
    _status_ok(C)


@pytest.mark.parametrize("V,start", [(1000, 0), (4096, 4096), (50257, 0)])
def test_cross_entropy_stats_and_grad(C, V, start):
    T = 64
    logits = bf(T, V, scale=3.0, seed=1)
    tgt = torch.randint(0, max(V, start + V), (T,), device="cuda")
    rm, se, tl = C.ce_stats(logits, tgt, start)
    rm_r, se_r, tl_r = ref.ce_stats(logits, tgt, start)
    torch.testing.assert_close(rm, rm_r, rtol=0, atol=0)
    torch.testing.assert_close(se, se_r, rtol=1e-3, atol=1e-3)
    torch.testing.assert_close(tl, tl_r, rtol=0, atol=0)
    lse = rm_r + torch.log(se_r)
    want = ref.ce_grad_(logits.clone(), tgt, lse, 0.25, start)
    got = logits.clone()
    C.ce_grad_(got, tgt, lse, 0.25, start)
    torch.testing.assert_close(got.float(), want.float(), rtol=2e-2, atol=1e-4)


def test_accumulate_add_merge(C):
    acc = torch.randn(1000 * 8 + 3, device="cuda")
    g = bf(1000 * 8 + 3, seed=1)
    want = acc + g.float()
    C.accumulate_(acc, g)
    torch.testing.assert_close(acc, want)
    a, b = bf(33, 200, seed=2), bf(33, 200, seed=3)
    torch.testing.assert_close(C.add(a, b).float(), (a.float() + b.float()).to(torch.bfloat16).float())
    B, S, h, d = 2, 20, 3, 64
    out, lse = torch.randn(B, S, h, d, device="cuda"), torch.randn(B, h, S, device="cuda")
    bo, bl = bf(B, S, h, d, seed=4), torch.randn(B, h, S, device="cuda")
    o_ref, l_ref = ref.merge_attention_(out.clone(), lse.clone(), bo, bl)
    C.merge_attention_(out, lse, bo, bl)
    torch.testing.assert_close(out, o_ref, rtol=1e-4, atol=1e-4)
    torch.testing.assert_close(lse, l_ref, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("master", [True, False])
def test_adamw_multi_tensor(C, master):
    torch.manual_seed(0)
    shapes = [(300, 64), (17,), (70000,), (128, 256)] * 8
    params = [torch.randn(*s, device="cuda").to(torch.bfloat16) for s in shapes]
    grads = [torch.randn(*s, device="cuda") for s in shapes]
    ms = [torch.zeros(*s, device="cuda") for s in shapes]
    vs = [torch.zeros(*s, device="cuda") for s in shapes]
    masters = [p.float().clone() if master else None for p in params]
    rp, rm, rv = [p.clone() for p in params], [m.clone() for m in ms], [v.clone() for v in vs]
    rmw = [m.clone() if m is not None else None for m in masters]
    for step in (1, 2):
        C.adamw_multi_(params, grads, ms, vs, masters, step, 1e-2, 0.9, 0.999, 1e-8, 0.01)
        ref.adamw_step_(rp, grads, rm, rv, rmw, step, 1e-2, 0.9, 0.999, 1e-8, 0.01)
    for a, b in zip(params, rp):
        torch.testing.assert_close(a.float(), b.float(), rtol=1e-2, atol=1e-2)
    for a, b in zip(ms, rm):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-6)
    if master:
        for a, b in zip(masters, rmw):
            torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("dtype,offset,count", [(torch.bfloat16, 0, 3), (torch.bfloat16, 1, 3), (torch.float32, 0, 3),
                                                (torch.float32, 1, 3), (torch.bfloat16, 0, 300)])
def test_adamw_chunk_edges_alignment_and_table_size(C, dtype, offset, count):
    """Sizes around a block's 4096 elements, slices that start off a 16-byte boundary, more tensors than one launch takes."""
    g = torch.Generator(device="cuda").manual_seed(5)
    sizes = [(1, 4095, 4096, 4097, 12289, 5)[i % 6] for i in range(2 * count)]
    new = lambda n, dt: torch.randn(n + offset, device="cuda", generator=g).to(dt)[offset:]
    params, grads = [new(n, dtype) for n in sizes], [new(n, torch.float32) for n in sizes]
    ms, vs = [new(n, torch.float32) for n in sizes], [new(n, torch.float32).abs() for n in sizes]
    masters = [None] * len(sizes)
    want = [x.clone() for x in params], [x.clone() for x in ms], [x.clone() for x in vs]
    C.adamw_multi_(params, grads, ms, vs, masters, 3, 1e-2, 0.9, 0.999, 1e-8, 0.01)
    ref.adamw_step_(want[0], grads, want[1], want[2], masters, 3, 1e-2, 0.9, 0.999, 1e-8, 0.01)
    # fp32 arithmetic in another order: a few ulps; a bf16 weight may round to its other neighbour, and
    # neighbours (8 significant bits) are between 2^-8 and 2^-7 of their value apart
    tol = dict(rtol=2 ** -7, atol=1e-6) if dtype == torch.bfloat16 else dict(rtol=1e-5, atol=1e-5)
    for got, exp, t in ((params, want[0], tol), (ms, want[1], dict(rtol=1e-5, atol=1e-6)), (vs, want[2], dict(rtol=1e-5, atol=1e-6))):
        for a, b in zip(got, exp):
            torch.testing.assert_close(a, b, **t)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("master", [False, True])
def test_adamw_does_not_depend_on_an_elements_place(C, dtype, master):
    """The same 2048 elements in a whole chunk (16-byte accesses), in a tensor's last chunk and off the alignment: equal bits."""
    g = torch.Generator(device="cuda").manual_seed(9)
    draw = lambda scale: torch.randn(2048, device="cuda", generator=g) * scale
    p, grad, m, v, w = draw(1.0).to(dtype), draw(1e-3), draw(1e-3), draw(1e-3) ** 2, draw(1.0)
    place = lambda x, off: torch.cat([x.new_zeros(off), x, x, x])[off:]
    results = []
    for off in (0, 1):
        t = [place(x, off) for x in (p, grad, m, v, w)]
        C.adamw_multi_([t[0]], [t[1]], [t[2]], [t[3]], [t[4] if master else None], 3, 1e-3, 0.9, 0.999, 1e-8, 0.01)
        results += [[x[i:i + 2048] for x in t] for i in (0, 2048, 4096)]
    for r in results[1:]:
        for a, b in zip(results[0], r):
            assert torch.equal(a, b)


@pytest.mark.parametrize("n", [1, 8191, 8192, 8193, 40000])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("c", [0.37, 1.0])
def test_scale_by_a_device_coefficient(C, n, offset, c):
    x = torch.randn(n + offset + 3, device="cuda")
    want = x.clone()
    want[offset:offset + n] *= c
    C.scale_(x[offset:offset + n], torch.tensor(c, device="cuda"))
    assert torch.equal(x, want)


@pytest.mark.parametrize("T", [1, 128, 255, 257, 600])
@pytest.mark.parametrize("H,I,hq,hkv,d", [(64, 128, 1, 1, 64), (192, 384, 3, 1, 64), (520, 640, 4, 2, 64), (256, 128, 2, 1, 128)])
def test_gemm_narrow_tiles_equal_wide_tiles(T, H, I, hq, hkv, d):
    """128-column against 256-column output tiles: the same products summed in the same order, whatever the tile and epilogue."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    x, a, gu = bf(T, H, seed=1), bf(T, I, seed=2), bf(T, 2 * I, seed=3)
    wq, wgu, wd = bf((hq + 2 * hkv) * d, H, seed=4), bf(2 * I, H, seed=5), bf(H, I, seed=6)
    cos, sin = ref.rope_tables(max(T, 8), d, 10000.0, device="cuda")
    results = []
    try:
        for n in (128, 256, 0):
            C.set_gemm_tile_n(n)
            results.append([C.gemm(x, wq, False, False), C.gemm(gu, wgu, False, True), C.gemm(a, wd, False, False),
                            C.gemm_rope(x, wq, cos, sin, hq + hkv, d, T), *C.gemm_swiglu(x, wgu), C.gemm_add(a, wd, x),
                            C.gemm_dgrad_swiglu_bwd(x, wd, gu)])
    finally:
        C.set_gemm_tile_n(0)
    _status_ok(C)
    torch.testing.assert_close(results[0][0].float(), x.float() @ wq.float().t(), rtol=2e-2, atol=2e-2 * math.sqrt(H))
    for other in results[1:]:
        for got, want in zip(results[0], other):
            assert torch.equal(got, want)


@pytest.mark.parametrize("T,N,K", [(64, 576, 49152), (2048, 576, 49160), (500, 520, 16392), (512, 2048, 16384), (1, 8, 8200)])
@pytest.mark.parametrize("into", [False, True])
def test_gemm_input_gradient_with_k_split(C, T, N, K, into):
    """Few output tiles behind a long K: parts of K are summed in an fp32 workspace and rounded once; also into rows of a wider
    output, whose other columns stay as they were."""
    from picotron_b200.ops import _ext
    C = _ext.load()
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    dy, w = bf(T, K, seed=1, scale=0.1), bf(K, N, seed=2, scale=0.1)
    big = torch.full((T, N + 16), 3.0, device="cuda", dtype=torch.bfloat16)
    out = big[:, 8:8 + N] if into else None
    n0 = C.launch_count()
    y = C.gemm(dy, w, False, True, out, False)
    assert C.launch_count() - n0 == 3, "this shape should be split"
    _status_ok(C)
    want = dy.double() @ w.double()
    # fp32 sums in another order (2^-24 sqrt(K) of sums of size sqrt(K)), then one rounding to bf16 (2^-9)
    assert _rel(y, want) < 2.5e-3
    if into:
        assert torch.equal(big[:, :8], torch.full_like(big[:, :8], 3.0)) and torch.equal(big[:, 8 + N:], torch.full_like(big[:, :8], 3.0))
    C.set_gemm_split_dgrad(False)
    try:
        assert _rel(C.gemm(dy, w, False, True), want) > 0.9 * _rel(y, want)       # no further off than the unsplit kernel
    finally:
        C.set_gemm_split_dgrad(True)


def test_gemm_switches_are_those_of_the_calling_thread(C):
    """A thread that switches the K split off for itself leaves the launches of the others as they were."""
    import threading
    C.set_gemm_pair(True)
    C.set_gemm_tma_epilogue(True)
    dy, w = bf(64, 49152, seed=1, scale=0.1), bf(49152, 576, seed=2, scale=0.1)

    def launches():
        n0 = C.launch_count()
        C.gemm(dy, w, False, True)
        return C.launch_count() - n0

    counts = [launches()]
    switched, looked = threading.Event(), threading.Event()

    def other():
        C.set_gemm_split_dgrad(False)
        counts.append(launches())
        switched.set()
        looked.wait(60)
        C.set_gemm_split_dgrad(True)

    t = threading.Thread(target=other)
    t.start()
    switched.wait(60)
    counts.append(launches())
    looked.set()
    t.join()
    _status_ok(C)
    assert counts[0] == counts[2] > counts[1] == 1
