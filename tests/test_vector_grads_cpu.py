"""Readiness of parameters whose gradients kernels add to the fp32 buffer, with the kernels stood in for on CPU ranks."""
import torch

from dist_utils import run_distributed


def _shared_vector_worker(rank, world):
    from teletron_b200.ops import _lib
    from teletron_b200.parallel.ddp import DistributedOptimizer, ParamBuffer
    import torch.distributed as dist

    class Shift(torch.autograd.Function):
        """x + v; the gradient of v goes into its buffer where it may."""

        @staticmethod
        def forward(ctx, x, v):
            ctx.v = v
            return x + v

        @staticmethod
        def backward(ctx, dy):
            mg, dv = _lib.main_grad_target(ctx.v, ctx.next_functions[1]), dy.sum(0)
            if mg is None:
                return dy, dv
            assert not fired()
            mg.add_(dv)
            _lib.grad_written(ctx.v)
            return dy, None

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.v = torch.nn.Parameter(torch.ones(8))
            self.out = torch.nn.Linear(8, 8, bias=False)

        def forward(self, x):           # v twice in one pass
            return self.out(Shift.apply(Shift.apply(x, self.v), self.v))

    torch.manual_seed(0)
    net = Net()
    buf = ParamBuffer(net, shard_world=1)
    opt = DistributedOptimizer(buf, dist.group.WORLD, overlap=True)
    bucket = buf.param_buckets["v"][0]
    fired = lambda: opt._fired[bucket]  # noqa: E731
    opt.begin_last_microbatch()
    x = torch.randn(4, 8) + rank
    net(x).square().sum().backward()
    assert fired()                                       # complete, so under way before the step
    opt.reduce_gradients()
    total = net.v.main_grad.clone()
    x2 = x.clone().requires_grad_()
    net(x2).square().sum().backward(inputs=[x2])
    mine = 2 * x2.grad.sum(0)
    dist.all_reduce(mine)
    return total, mine


def test_vector_used_twice_reports_once_after_both_uses():
    for total, mine in run_distributed(_shared_vector_worker, 2):
        torch.testing.assert_close(total, mine)
