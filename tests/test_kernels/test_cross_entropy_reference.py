"""The torch form of the cross-entropy statistics (CPU tensors, and logits that the kernels do not take): rows without a finite
column in a shard, as masked logits leave them."""
import pytest
import torch
import torch.distributed as dist
import torch.nn.functional as F

import colossalai_b200
from colossalai_b200.ops import cross_entropy as ce
from colossalai_b200.shardformer.layer import cross_entropy_1d, dist_log_prob_1d
from colossalai_b200.testing import rerun_if_address_is_in_use, spawn


@pytest.mark.parametrize("valid", [0, 5, 8])
def test_row_stats_of_masked_rows(valid):
    torch.manual_seed(0)
    x = torch.randn(4, 8)
    x[1] = torch.finfo(torch.float32).min
    x[2] = float("-inf")
    x[3] = float("-inf")
    x[3, 2] = 1.0
    m, s, t = ce.row_stats(x, torch.full((4,), 2), 0, -100, valid)
    if valid == 0:
        assert torch.isneginf(m).all() and not s.any() and not t.any()
        return
    x64 = x[:, :valid].double()
    rows = [0, 1, 3]
    assert torch.equal(m[rows], x[rows, :valid].max(-1).values) and torch.isneginf(m[2]) and s[2] == 0
    torch.testing.assert_close(s[rows].double(), (x64 - x64.max(-1, keepdim=True).values).exp().sum(-1)[rows], rtol=1e-6, atol=0)
    assert torch.equal(t, x[:, 2])
    # against the maximum over all shards: a shard without a finite column adds nothing
    assert ce.rescale(torch.stack([m, s, t]), torch.full((4,), 2.0))[0][2] == 0


def _shards(rank, world_size, port):
    colossalai_b200.launch(rank, world_size, "127.0.0.1", port, backend="gloo", verbose=False)
    torch.manual_seed(0)
    full = torch.randn(6, 16)
    full[1, 8:] = full[4, 8:] = float("-inf")                    # every column of the second shard
    full[2, :8] = float("-inf")                                  # of the first
    labels = torch.tensor([3, 5, 9, -100, 0, 15])
    want = full.clone().requires_grad_()
    ref = F.cross_entropy(want, labels, ignore_index=-100)
    ref.backward()
    mine = full.chunk(world_size, -1)[rank].clone().requires_grad_()
    loss = cross_entropy_1d(mine, labels, process_group=None)
    loss.backward()
    torch.testing.assert_close(loss, ref, rtol=1e-6, atol=1e-6)
    torch.testing.assert_close(mine.grad, want.grad.chunk(world_size, -1)[rank], rtol=1e-5, atol=1e-7)
    lp = dist_log_prob_1d(mine.detach(), labels.clamp(min=0), process_group=None)
    want_lp = F.log_softmax(full, -1).gather(-1, labels.clamp(min=0)[:, None]).reshape(lp.shape)
    torch.testing.assert_close(lp, want_lp, rtol=1e-6, atol=1e-6)
    dist.barrier()
    dist.destroy_process_group()


@rerun_if_address_is_in_use()
def test_vocab_shards_without_a_finite_column():
    spawn(_shards, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("V", [8, 1000, 4096, 16384, 16392, 20488])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gradient_of_rows_without_a_label(V, dtype):
    """Zero where every logit is finite (or minus infinity beside finite ones) and NaN where the exponentials against the row's maximum
    are not numbers, between rows with labels; sizes on and beside what a block's threads hold at a time."""
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(8, V, device="cuda", generator=g).to(dtype)
    x[1, 3], x[2, 5], x[4, 2], x[6] = float("nan"), float("inf"), -float("inf"), -float("inf")
    labels = torch.full((8,), -100, device="cuda")
    labels[0], labels[7], labels[5] = V - 1, 0, 2
    z = x.clone().requires_grad_(True)
    (grad,) = torch.autograd.grad(cross_entropy_1d(z, labels, process_group="local"), z)
    top = torch.where(x.isnan(), -float("inf"), x).amax(-1, keepdim=True).double()
    want = (x.double() - top).exp() * 0.0
    keep = labels >= 0
    want[keep] = (x[keep].double().softmax(-1) - torch.nn.functional.one_hot(labels[keep], V)) / 3
    assert torch.equal(grad.isnan(), want.isnan()) and int(grad.isnan().sum()) == V + 2
    # a rounding to the type, and of the exponential and the sum in fp32
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    assert ((grad.double() - want).abs()[~want.isnan()] <= unit * want.abs()[~want.isnan()] + 1e-9).all()
    assert not grad[3].any() and not grad[4].any()
