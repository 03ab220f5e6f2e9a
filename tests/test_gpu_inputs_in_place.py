"""One rank: inputs are read where the caller keeps them.  Inputs that cannot be (misaligned, or lying in a buffer that the
call writes) still go through the workspace, with bitwise the same results, and no input is changed."""
import pytest
import torch


pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mxfp8", [False, True])
def test_awkward_inputs_give_the_same_results(dist_ctx, mxfp8):
    import torch.distributed as dist
    import mok
    F, dev = mok.functional, torch.device("cuda", torch.cuda.current_device())
    T, H, I, E, K = 768, 512, 256, 6, 2
    g = torch.Generator(device=dev).manual_seed(4)
    normal = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.bfloat16)  # noqa: E731
    config = F.MoKConfig(macrobatch_size=8192, schedule_capacity_multiplier=3.0)
    ws = F.create_workspace(config, dist.group.WORLD, device=dev, num_local_tokens=T, hidden_size=H, topk=K)
    x, dy, rw = normal(T, H), normal(T, H), torch.rand(T, K, generator=g, device=dev) + 0.1
    routes = torch.topk(torch.randn(T, E, generator=g, device=dev), K).indices
    shared = [normal(I, H) * 0.05, normal(I, H) * 0.05, normal(H, I) * 0.05]
    routed = [normal(E, I, H) * 0.05, normal(E, I, H) * 0.05, normal(E, H, I) * 0.05]
    back = routed
    if mxfp8:
        q = mok.quantize_routed_weights(*routed)
        routed, back = (q[0][:2], q[1][:2], q[2][:2]), (q[0], q[1], q[2][2:])

    def run(x_, dy_of, rw_, rw_of=None):
        sched = F.build_schedule(ws, config, routes, num_local_experts=E)
        out, ctx = F.forward(config, ws, sched, x_, rw_, *shared, *routed)
        if rw_of is not None:
            rw_ = rw_of()
        grads = F.backward(config, ws, sched, ctx, dy_of(), x_, rw_, *shared, *back)
        torch.cuda.synchronize()
        mok.ops.check_status(dev)
        return [out, *grads]

    def misaligned(t):
        flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=dev)[1:]
        flat.copy_(t.flatten())
        return flat.view(t.shape)

    def inside(buffer, t):
        view = buffer.flatten()[:t.numel()].view(t.shape)
        view.copy_(t)
        return view

    before = [t.clone() for t in (x, dy, rw)]
    want = run(x, lambda: dy, rw)
    for a, b in zip(before, (x, dy, rw)):
        assert torch.equal(a, b)
    assert misaligned(x).data_ptr() % 16 != 0
    for got in (run(misaligned(x), lambda: misaligned(dy), misaligned(rw)),
                run(x, lambda: inside(ws.d_x_routed_buffer, dy), rw, lambda: inside(ws.d_router_weight_buffer, rw))):
        for i, (a, b) in enumerate(zip(want, got)):
            assert torch.equal(a, b), i


def test_traced_layer_reads_the_inputs_of_the_replay(dist_ctx):
    """make_fx with real tensors records the ops and their address lists; the graph must work on other inputs."""
    import torch.distributed as dist
    import mok
    from torch.fx.experimental.proxy_tensor import make_fx
    F, dev = mok.functional, torch.device("cuda", torch.cuda.current_device())
    T, H, I, E, K = 512, 256, 256, 4, 2
    g = torch.Generator(device=dev).manual_seed(6)
    normal = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.bfloat16)  # noqa: E731
    config = F.MoKConfig(macrobatch_size=4096, schedule_capacity_multiplier=3.0)
    ws = F.create_workspace(config, dist.group.WORLD, device=dev, num_local_tokens=T, hidden_size=H, topk=K)
    routes = torch.topk(torch.randn(T, E, generator=g, device=dev), K).indices
    w = [normal(I, H) * 0.05, normal(I, H) * 0.05, normal(H, I) * 0.05, normal(E, I, H) * 0.05, normal(E, I, H) * 0.05, normal(E, H, I) * 0.05]
    sched = F.build_schedule(ws, config, routes, num_local_experts=E)

    def layer(x, rw, dy):
        out, ctx = F.forward(config, ws, sched, x, rw, *w)
        return (out, *F.backward(config, ws, sched, ctx, dy, x, rw, *w))

    first, second = [(normal(T, H), torch.rand(T, K, generator=g, device=dev) + 0.1, normal(T, H)) for _ in range(2)]
    graph = make_fx(layer)(*first)
    want = [t.clone() for t in layer(*second)]
    for i, (a, b) in enumerate(zip(want, graph(*second))):
        assert a.float().abs().sum() > 0 and torch.equal(a, b), i
    mok.ops.check_status(dev)
