"""Parallel strategies on real GPUs (bf16, NCCL, CUDA kernels) against the fp32 CPU oracle."""
import pytest
import torch

from dist_utils import run_distributed
import parallel_harness as H

pytestmark = [pytest.mark.gpu, pytest.mark.multigpu]


def _run(tp=1, cp=1, pp=1, dp=1, engine="1f1b", grad_acc=2, layers=4, graph=False, cp_layout=None):
    world = tp * cp * pp * dp
    if torch.cuda.device_count() < world:
        pytest.skip(f"needs {world} GPUs")
    res = run_distributed(H.worker, world, tp, cp, pp, dp, engine, grad_acc, layers, True, graph, None, cp_layout,
                          backend="nccl")
    H.check(res, tp, cp, pp, dp, grad_acc, layers, gpu=True)


def test_ops_on_a_second_device_of_the_process():
    """Large shared memory has to be opted into on each device."""
    from picotron_b200 import ops
    from picotron_b200.ops import reference as ref
    for dev in ("cuda:0", "cuda:1"):
        g = torch.Generator(device=dev).manual_seed(1)
        x, dy = (torch.randn(256, 2048, device=dev, generator=g).to(torch.bfloat16) for _ in range(2))
        w, rstd, acc = x[0].contiguous(), torch.ones(256, device=dev), torch.zeros(2048, device=dev)
        dx, _ = ops.rmsnorm_bwd(dy, x, w, rstd, None, acc)
        want, _ = ref.rmsnorm_bwd(dy, x, w, rstd, None)
        torch.testing.assert_close(dx.float(), want.float(), rtol=2 ** -7, atol=1e-2)      # one bf16 rounding of fp32 terms
        y, want = ops.linear_fwd(x, dy).double(), x.double() @ dy.double().t()
        assert float((y - want).norm() / want.norm()) < 4e-3                               # one bf16 rounding
        q, do = x.view(1, 256, 32, 64), dy.view(1, 256, 32, 64)
        o, lse = ops.attention_fwd(q, q, q, True)
        o_ref, lse_ref = ref.attention_fwd(q, q, q, True, 0.125)
        torch.testing.assert_close(o.float(), o_ref.float(), rtol=2e-2, atol=2e-2)
        for got, want in zip(ops.attention_bwd(do, q, q, q, o, lse, True), ref.attention_bwd(do, q, q, q, o_ref, lse_ref, True, 0.125)):
            assert float((got.float() - want.float()).norm() / want.float().norm()) < 2e-2


def test_dp2():
    _run(dp=2)


def test_tp2():
    _run(tp=2)


def test_pp2_1f1b():
    _run(pp=2, grad_acc=3)


def test_pp2_afab():
    _run(pp=2, engine="afab", grad_acc=3)


def test_cp2():
    _run(cp=2)


def test_dp2_tp2():
    _run(dp=2, tp=2)


def test_tp2_cp2_pp2():
    _run(tp=2, cp=2, pp=2)


def test_dp2_tp2_pp2():
    _run(dp=2, tp=2, pp=2)


def test_tp2_micro_batches_replayed_from_a_cuda_graph():
    _run(tp=2, grad_acc=3, graph=True)


def test_cp2_micro_batches_replayed_from_a_cuda_graph():
    _run(cp=2, grad_acc=3, graph=True)


def test_dp2_micro_batches_replayed_from_a_cuda_graph():
    _run(dp=2, grad_acc=3, graph=True)


def test_cp2_zigzag_layout():
    _run(cp=2, cp_layout="zigzag")
