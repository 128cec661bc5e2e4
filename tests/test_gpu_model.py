"""The fused model on the GPU (bf16, CUDA kernels) against the same model on CPU (fp32, PyTorch restatements)."""
import contextlib
import threading

import pytest
import torch

from picotron_b200.config import ModelConfig
from picotron_b200.models.llama import Llama
from picotron_b200.optim import FusedAdamW
from picotron_b200.parallel.data_parallel import DataParallelBucket

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,d", [(8, 8, 64), (8, 2, 64), (4, 2, 128)])
def test_model_loss_and_grads_match_cpu_fp32(hq, hkv, d):
    from picotron_b200.ops import _ext
    C = _ext.load()
    torch.manual_seed(0)
    cfg = ModelConfig(hidden_size=hq * d, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=hq,
                      num_key_value_heads=hkv, vocab_size=1024, max_position_embeddings=256)
    cpu = Llama(cfg, init="normal")
    gpu = Llama(cfg, init="normal")
    gpu.load_state_dict(cpu.state_dict())
    gpu = gpu.to(torch.bfloat16).cuda()
    with torch.no_grad():                      # same (bf16-rounded) weights on both sides
        for pc, pg in zip(cpu.parameters(), gpu.parameters()):
            pc.copy_(pg.float().cpu())
    wg = DataParallelBucket(gpu)
    ids = torch.randint(0, cfg.vocab_size, (2, 256))
    tgt = torch.randint(0, cfg.vocab_size, (2, 256))
    n0 = C.launch_count()
    loss_g = wg(input_ids=ids.cuda(), target_ids=tgt.cuda())
    loss_g.backward()
    torch.cuda.synchronize()
    assert C.launch_count() > n0, "the CUDA kernels did not run"
    assert C.kernel_status() == 0
    loss_c = cpu(ids, target_ids=tgt)
    loss_c.backward()
    assert abs(loss_g.item() - loss_c.item()) < 3e-2, (loss_g.item(), loss_c.item())
    for (n, pc), pg in zip(cpu.named_parameters(), gpu.parameters()):
        g, r = pg.main_grad.float().cpu(), pc.grad
        err = (g - r).norm() / (r.norm() + 1e-12)
        assert err < 5e-2, f"{n}: relative gradient error {err:.4f}"
    opt = FusedAdamW(wg.parameters(), lr=1e-3)
    before = [p.detach().clone() for p in gpu.parameters()]
    opt.step()
    wg.reset()
    torch.cuda.synchronize()
    assert any(not torch.equal(a, b) for a, b in zip(before, gpu.parameters()))
    assert all(torch.isfinite(p).all() for p in gpu.parameters())


@pytest.mark.parametrize("hq,hkv,d,inter,seq", [(4, 4, 64, 512, 130), (6, 2, 64, 320, 97), (2, 1, 128, 192, 256), (4, 2, 64, 200, 64)])
@pytest.mark.parametrize("wrapped", [True, False])
def test_native_layer_matches_the_separate_calls(monkeypatch, hq, hkv, d, inter, seq, wrapped):
    """The same kernels in the same order: equal outputs, and gradients equal up to the order of the atomic dQ sums; with widths
    that the fused epilogues do not cover, and without gradient buckets (autograd gradients keep the separate calls)."""
    from picotron_b200 import ops
    torch.manual_seed(1)
    cfg = ModelConfig(hidden_size=hq * d, intermediate_size=inter, num_hidden_layers=2, num_attention_heads=hq,
                      num_key_value_heads=hkv, vocab_size=256, max_position_embeddings=seq + 5)
    model = Llama(cfg, init="normal").to(torch.bfloat16).cuda()
    run = DataParallelBucket(model) if wrapped else model
    ids = torch.randint(0, cfg.vocab_size, (2, seq), device="cuda")
    results = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(ops, "runs_layer_natively", lambda x: False)
        if wrapped:
            run.reset()
        else:
            model.zero_grad()
        with torch.no_grad():
            logits = model(ids)
        loss = run(input_ids=ids, target_ids=ids.roll(-1, 1))
        loss.backward()
        results.append((logits, loss.detach(), [(p.main_grad if wrapped else p.grad).float().clone() for p in model.parameters()]))
    (la, a, ga), (lb, b, gb) = results
    assert torch.equal(la, lb) and torch.equal(a, b)
    for x, y in zip(ga, gb):
        # dQ is summed in fp32 in any order and rounded to bf16: neighbours (2^-8) in places, carried through two layers
        assert float((x - y).norm()) <= 4 * 2 ** -8 * float(y.norm()) + 1e-6


@pytest.mark.parametrize("hq,hkv,d,inter,B,S", [(4, 2, 64, 320, 2, 97), (2, 1, 128, 200, 1, 64)])
def test_layer_ops_with_a_tensor_per_activation(hq, hkv, d, inter, B, S):
    """``ops.decoder_layer_fwd`` hands every activation out, and ``ops.decoder_layer_bwd`` takes such a list, wherever its tensors
    lie; both equal the calls that keep them in two allocations."""
    from picotron_b200 import ops
    H, Q, T = hq * d, (hq + 2 * hkv) * d, B * S
    g = torch.Generator(device="cuda").manual_seed(3)
    bf = lambda *s: (0.05 * torch.randn(*s, device="cuda", generator=g)).to(torch.bfloat16)
    x, dout, ln1, ln2 = 20 * bf(T, H), 20 * bf(T, H), 1 + bf(H), 1 + bf(H)
    w_qkv, wo, w_gu, wd = bf(Q, H), bf(H, H), bf(2 * inter, H), bf(H, inter)
    angles = torch.rand(S, d // 2, device="cuda", generator=g)
    cos, sin, scale = angles.cos(), angles.sin(), d ** -0.5
    fwd = (x, ln1, w_qkv, cos, sin, wo, ln2, w_gu, wd, 1e-5, B, S, hq, hkv, d, scale)
    out, h1, rstd1, qkv, o, lse, x_mid, rstd2, h2, gu, a = ops.decoder_layer_fwd(*fwd)
    packed = ops.decoder_layer_fwd_packed(*fwd)
    saved = [x, rstd1, h1, qkv, o, lse, x_mid, rstd2, h2, gu, a]
    assert torch.equal(out, packed[0])
    for mine, theirs in zip(saved[1:], ops.decoder_layer_saved(packed[1], packed[2], B, S, H, inter, hq, hkv, d)):
        assert mine.shape == theirs.shape and torch.equal(mine, theirs)
    assert [tuple(t.shape) for t in saved] == [(T, H), (T,), (T, H), (T, Q), (T, H), (B, hq, S), (T, H), (T,), (T, H), (T, 2 * inter), (T, inter)]

    def regions():
        flat = torch.zeros(Q * H + H * H + 3 * inter * H + 2 * H, device="cuda")
        shapes = [(hq * d, H), (hkv * d, H), (hkv * d, H), (H, H), (inter, H), (inter, H), (H, inter), (H,), (H,)]
        return list(t.view(s) for t, s in zip(flat.split([torch.Size(s).numel() for s in shapes]), shapes)), flat

    rest = (ln1, w_qkv, cos, sin, wo, ln2, w_gu, wd)
    mg, flat = regions()
    dx = ops.decoder_layer_bwd_packed(dout, x, packed[1], packed[2], *rest, mg, B, S, hq, hkv, d, scale)
    mg2, flat2 = regions()
    dx2 = ops.decoder_layer_bwd(dout, [t.clone() for t in saved], *rest, mg2, B, S, hq, hkv, d, scale)
    # one key block: dQ is not added up in any order; the norm weights' gradients are, over T rows in fp32
    assert torch.equal(dx, dx2)
    torch.testing.assert_close(flat, flat2, rtol=1e-4, atol=1e-5)
    with pytest.raises(RuntimeError):
        ops.decoder_layer_bwd(dout, [t.clone() for t in saved[:9]] + [gu[:, 1:], a], *rest, mg2, B, S, hq, hkv, d, scale)


def test_checked_mode_sees_a_loss_that_is_not_finite_without_a_gradient():
    from picotron_b200 import ops
    x, w = torch.ones(3, 64, device="cuda", dtype=torch.bfloat16), torch.ones(16, 64, device="cuda", dtype=torch.bfloat16)
    targets, terms = torch.zeros(3, device="cuda", dtype=torch.long), torch.empty(3, device="cuda")
    ops.enable_checked_mode(True)
    try:
        ops.linear_ce_loss(x, w, targets, 0, 1.0, terms, False)
        x[1, 2] = float("nan")
        with pytest.raises(FloatingPointError, match="linear_ce_loss"):
            ops.linear_ce_loss(x, w, targets, 0, 1.0, terms, False)
    finally:
        ops.enable_checked_mode(False)


@pytest.mark.parametrize("layers,hq,hkv,d,inter,B,S", [(1, 2, 1, 64, 192, 1, 1), (3, 3, 1, 64, 320, 2, 97), (2, 2, 2, 128, 200, 1, 130)])
def test_layers_in_one_native_call_equal_the_layers_one_by_one(layers, hq, hkv, d, inter, B, S):
    """The same launches: outputs, losses and logits equal to the bit, gradients up to the order of atomic additions; a hook on a layer is still
    called, saved-tensor hooks get the tensors of one layer after the other (the layers run one by one then); weights that do not lie
    side by side are no matter; another layer's norm weight swapped for the call is used."""
    from picotron_b200.models import llama as M
    torch.manual_seed(2)
    cfg = ModelConfig(hidden_size=hq * d, intermediate_size=inter, num_hidden_layers=layers, num_attention_heads=hq,
                      num_key_value_heads=hkv, vocab_size=256, max_position_embeddings=S + 3)
    model = Llama(cfg, init="normal").to(torch.bfloat16).cuda()
    w = model.decoder_layers[-1].mlp.up_proj.weight
    w.data = w.data.clone()                                     # no longer behind its gate projection
    ids = torch.randint(0, cfg.vocab_size, (B, S), device="cuda")
    stacks = []
    one_call = M._run_stack

    def watched(*a):
        y = one_call(*a)
        stacks.append(y is not None)
        return y

    def passes(**swap):
        call = lambda **kw: torch.func.functional_call(model, swap, (ids,), kw) if swap else model(ids, **kw)   # noqa: E731
        out = []
        with torch.no_grad():
            out += [call(), call(target_ids=ids)]
        with torch.inference_mode():
            out.append(call())
        return out

    M._run_stack = watched
    try:
        passes()                                                # (the layers put their packed weights together)
        stacks.clear()
        together, swapped = passes(), passes(**{"final_norm.weight": model.final_norm.weight * 2,
                                                "decoder_layers.0.input_layernorm.weight": model.decoder_layers[0].input_layernorm.weight * 2})
        assert stacks == [True] * 6
        model.embedding.weight.requires_grad_(layers != 2)      # once with an input that needs no gradient
        wrapped = DataParallelBucket(model)

        def grads(hooked, offload=False):
            wrapped.reset()
            stacks.clear()
            calls = []
            handle = model.decoder_layers[0].register_forward_hook(lambda *a: calls.append(1)) if hooked else None
            with torch.autograd.graph.save_on_cpu() if offload else contextlib.nullcontext():
                loss = wrapped(ids, target_ids=ids)
            loss.backward()
            if hooked:
                handle.remove()
            assert stacks == [not hooked and not offload] and len(calls) == hooked
            return [loss.detach().clone()] + [p.main_grad.clone() for p in model.parameters() if p.requires_grad]

        many, each, offloaded = grads(False), grads(True), grads(False, True)
        handles = [layer.register_forward_pre_hook(lambda *a: None) for layer in model.decoder_layers]
        stacks.clear()
        single, single_swapped = passes(), passes(**{"final_norm.weight": model.final_norm.weight * 2,
                                                     "decoder_layers.0.input_layernorm.weight": model.decoder_layers[0].input_layernorm.weight * 2})
        assert stacks == [False] * 6
        for h in handles:
            h.remove()
    finally:
        M._run_stack = one_call
    for x, y in zip(together + swapped, single + single_swapped):
        assert torch.equal(x, y)
    assert not torch.equal(together[0], swapped[0])
    assert torch.equal(many[0], each[0]) and torch.equal(offloaded[0], each[0])
    for x, y in zip(many[1:] + offloaded[1:], each[1:] + each[1:]):
        # (dQ of more than two key blocks and the norm and embedding gradients add in any order: fp32 sums, rounded to bf16 once)
        assert float((x - y).norm()) <= 4e-3 * float(y.norm()) + 1e-12


@pytest.mark.parametrize("layers,T,H,I", [(1, 64, 192, 384), (4, 64, 192, 384), (4, 700, 192, 384), (2, 64, 1536, 1600)])
def test_weights_changed_just_before_a_pass_are_those_it_uses(layers, T, H, I):     # noqa: E741
    """The layers' GEMMs fetch weights and saved activations ahead of the kernel before them; what an optimizer step or a copy wrote right before
    the pass has to be seen, and a backward pass reads its own forward's activations: every pass equals the same one layer by layer. (Width
    1536: output and down projections and input gradients share K in clusters.)"""
    from picotron_b200.ops import _ext
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        for kind, n, k in (("fwd", H, H), ("add", H, I), ("dgrad", H, H), ("dgrad", H, 2 * I)):
            assert (_ext.load().gemm_plan(kind, T, n, k) == (128, -2)) == (H == 1536)
    torch.manual_seed(3)
    cfg = ModelConfig(hidden_size=H, intermediate_size=I, num_hidden_layers=layers, num_attention_heads=H // 64, num_key_value_heads=H // 192,
                      vocab_size=256, max_position_embeddings=T)
    model = Llama(cfg, init="normal").to(torch.bfloat16).cuda()
    wrapped = DataParallelBucket(model)
    opt = FusedAdamW(wrapped.parameters(), lr=2e-2)
    ids = torch.randint(0, cfg.vocab_size, (1, T), device="cuda")
    model(ids, target_ids=ids)                                  # (the layers put their packed weights together)
    start = [p.detach().clone() for p in model.parameters()]

    def train(hooked):
        with torch.no_grad():
            for p, q in zip(model.parameters(), start):
                p.copy_(q)
        opt.state.clear()
        wrapped.reset()
        handles = [layer.register_forward_pre_hook(lambda *a: None) for layer in model.decoder_layers] if hooked else []
        out = []
        for _ in range(4):
            loss = wrapped(ids, target_ids=ids)
            loss.backward()
            out += [loss.detach()] + [p.main_grad.clone() for p in model.decoder_layers[0].attention.parameters()]
            opt.step()
            wrapped.reset()
            with torch.no_grad():
                out.append(model(ids))                          # logits with the weights of this moment
        for h in handles:
            h.remove()
        return out

    together, single = train(False), train(True)
    assert float((together[-1] - together[5]).float().norm()) > 0.1 * float(together[5].float().norm()), "the weights hardly moved"
    for x, y in zip(together, single):
        # (gradients are summed in any order in places, and AdamW moves weights by what is left of them)
        assert float((x.float() - y.float()).norm()) <= 3e-2 * float(y.float().norm()) + 1e-12


@pytest.mark.parametrize("layers,inter,B", [(1, 1024, 2), (2, 1024, 2), (5, 1000, 2), (3, 1024, 48)])
def test_weight_gradients_on_a_second_stream(layers, inter, B):
    """Layers large enough that their weight gradients run beside their input gradients (12 GFLOP and more): the gradients of several micro-batches
    equal those layer by layer, on the default stream, on another one, from two threads at once, under saved-tensor hooks (layer by layer again),
    and from a captured graph that is replayed; memory that is freed right after the pass is not written by it any more. (48 x 1024 tokens: scratch beyond
    512 MiB, one area for all layers.)"""
    torch.manual_seed(4)
    cfg = ModelConfig(hidden_size=512, intermediate_size=inter, num_hidden_layers=layers, num_attention_heads=8, num_key_value_heads=4,
                      vocab_size=512, max_position_embeddings=1024)
    S = 1024

    def build():
        torch.manual_seed(5)
        model = Llama(cfg, init="normal").to(torch.bfloat16).cuda()
        return DataParallelBucket(model)

    g = torch.Generator(device="cuda").manual_seed(6)
    batches = [torch.randint(0, cfg.vocab_size, (B, S), device="cuda", generator=g) for _ in range(3)]

    def accumulate(w, context=None):
        w.reset()
        for i, ids in enumerate(batches):
            w.require_backward_grad_sync = i == len(batches) - 1
            with context() if context else contextlib.nullcontext():
                loss = w(input_ids=ids, target_ids=ids, loss_scale=0.5)
            loss.backward()
            # what the pass freed is taken and overwritten at once
            junk = [torch.full((n,), float("nan"), device="cuda") for n in (1 << 18, 1 << 20, 1 << 22)]
            del junk, loss
        return w.bucket_manager.flat

    def close(x, y):
        # (dQ, the norm weights' and the embedding's gradients add in any order; a rounding of bf16 moved by that moves what follows)
        assert torch.isfinite(x).all() and float((x - y).norm()) <= 4e-3 * float(y.norm())

    w = build()
    accumulate(w)
    handles = [layer.register_forward_pre_hook(lambda *a: None) for layer in w.module.decoder_layers]
    want = accumulate(w).clone()
    for h in handles:
        h.remove()
    close(accumulate(w), want)
    close(accumulate(w, torch.autograd.graph.save_on_cpu), want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        close(accumulate(w), want)
    torch.cuda.current_stream().wait_stream(side)

    models, errors = [build(), build()], []

    def work(m):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                accumulate(m)
                torch.cuda.current_stream().synchronize()
        except Exception as e:                               # noqa: BLE001
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(m,)) for m in models]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for m in models:
        close(m.bucket_manager.flat, want)

    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        w.require_backward_grad_sync = False
        w(input_ids=batches[0], target_ids=batches[0], loss_scale=0.5).backward()
    torch.cuda.current_stream().wait_stream(s)
    ids = batches[0].clone()
    with torch.cuda.graph(graph):
        w(input_ids=ids, target_ids=ids, loss_scale=0.5).backward()
    w.reset()
    for b in batches:
        ids.copy_(b)
        graph.replay()
    close(w.bucket_manager.flat, want)


def _side_stream_model():
    """Layers whose weight gradients run on a second stream (12 GFLOP and more), a batch, and the gradients layer by layer."""
    torch.manual_seed(7)
    cfg = ModelConfig(hidden_size=512, intermediate_size=1024, num_hidden_layers=3, num_attention_heads=8, num_key_value_heads=4,
                      vocab_size=512, max_position_embeddings=1024)
    w = DataParallelBucket(Llama(cfg, init="normal").to(torch.bfloat16).cuda())
    w.require_backward_grad_sync = False
    ids = torch.randint(0, cfg.vocab_size, (2, 1024), device="cuda")
    handles = [layer.register_forward_pre_hook(lambda *a: None) for layer in w.module.decoder_layers]
    w(input_ids=ids, target_ids=ids).backward()
    for h in handles:
        h.remove()
    want = w.bucket_manager.flat.clone()
    w.reset()
    return w, ids, want


@pytest.mark.parametrize("streams", [1, 6])
def test_eager_backward_while_another_thread_captures_one(streams):
    """Autograd runs the backward passes of both threads on one thread of its own: the captured one's second stream has to stay out of the eager
    ones, on one stream and on more than a thread keeps second streams for."""
    captured, eager = _side_stream_model(), [_side_stream_model() for _ in range(streams)]
    s, graph, errors = torch.cuda.Stream(), torch.cuda.CUDAGraph(), []
    others = [torch.cuda.Stream() for _ in eager]

    def one_pass(w, ids):
        w(input_ids=ids, target_ids=ids).backward()

    def work():
        try:
            for _ in range(2):
                for (w, ids, _), stream in zip(eager, others):
                    with torch.cuda.stream(stream):
                        w.reset()
                        one_pass(w, ids)
        except Exception as e:                               # noqa: BLE001
            errors.append(e)

    for stream in [s] + others:
        stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        one_pass(*captured[:2])
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        one_pass(*captured[:2])
        thread = threading.Thread(target=work)
        thread.start()
        thread.join()
        one_pass(*captured[:2])                              # (the capture goes on)
    assert not errors, errors
    captured[0].reset()
    graph.replay()
    torch.cuda.synchronize()
    for (w, _, want), passes in zip([captured] + eager, [2] + [1] * streams):
        got = w.bucket_manager.flat
        # (dQ, the norm weights' and the embedding's gradients add in any order; a rounding of bf16 moved by that moves what follows)
        assert torch.isfinite(got).all() and float((got - passes * want).norm()) <= 4e-3 * passes * float(want.norm())


@pytest.mark.parametrize("full", [False, True])
def test_memory_of_the_layers_backward(full):
    """What the backward pass takes beside what was there is within its plan; on a device too full for two streams' scratch it runs on one and
    takes what one stream takes."""
    from picotron_b200.utils.memory import plan_memory
    cfg = ModelConfig(hidden_size=512, intermediate_size=1024, num_hidden_layers=3, num_attention_heads=8, num_key_value_heads=4,
                      vocab_size=512, max_position_embeddings=1024)
    B, S = 16, 1024
    torch.manual_seed(8)
    w = DataParallelBucket(Llama(cfg, init="normal").to(torch.bfloat16).cuda())
    w.require_backward_grad_sync = False
    ids = torch.randint(0, cfg.vocab_size, (B, S), device="cuda")
    w(input_ids=ids, target_ids=ids).backward()
    want = w.bucket_manager.flat.clone()
    w.reset()
    loss = w(input_ids=ids, target_ids=ids)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    T, H = B * S, 512
    scratch_one = T * (max(4 * 1024, 2 * H + 2 * 1024 + 4 * H + 4 * 8) + 4 * H)
    scratch_two = 2 * T * (4 * 1024 + 2 * H + 2 * 1024 + 4 * H + 4 * 8 + 4 * H)
    others = 6 * T * H * 2 + (40 << 20)                         # gradients between layers and of the head; K-split workspaces
    total = torch.cuda.get_device_properties(0).total_memory
    assert scratch_one + others < scratch_two
    try:
        if full:
            torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + scratch_one + others) / total)
        loss.backward()
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    taken = torch.cuda.max_memory_allocated() - before
    planned = plan_memory(cfg, micro_batch_size=B, seq_length=S, fused_comm=False).bytes["transients"]
    assert taken < scratch_one + others if full else scratch_two < taken <= planned, (taken, planned)
    got = w.bucket_manager.flat
    # (dQ, the norm weights' and the embedding's gradients add in any order; a rounding of bf16 moved by that moves what follows)
    assert float((got - want).norm()) <= 4e-3 * float(want.norm())
