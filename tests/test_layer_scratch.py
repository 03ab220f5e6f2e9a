"""A layer call allocates the scratch that its kernels use and no more: which bf16 buffers and row sums that is, under every switch
(CPU), and the memory that the calls of one rank take beyond their outputs (GPU)."""
import pytest
import torch


def _args(T, K, E, ep=1, H=2048, I=2048):
    from mok import _native as nat
    a = nat.LayerArgs()
    a.ep_size, a.num_local_tokens, a.topk, a.num_local_experts, a.hidden, a.intermediate = ep, T, K, E, H, I
    return nat, a


@pytest.mark.parametrize("ep", [1, 2])
@pytest.mark.parametrize("env,act,grad", [({}, 0, 0), ({"MOK_NO_FUSED_EPILOGUE": "1"}, 1, 0), ({"MOK_NO_FUSED_ACT": "1"}, 1, 1)])
def test_scratch_of_the_mxfp8_calls(monkeypatch, ep, env, act, grad):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    nat, a = _args(512, 8, 16, ep)
    want = (nat.SCRATCH_DISPATCHED if ep > 1 else 0) + act * nat.SCRATCH_ACTIVATIONS + grad * nat.SCRATCH_GRADIENTS
    assert nat.lib().mok_layer_scratch(nat.ctypes.byref(a), 1) == want


@pytest.mark.parametrize("T,K,E,H,I,partials", [(768, 8, 64, 4096, 1024, True),      # 96 rows per expert
                                                (768, 8, 63, 4096, 1024, False),     # a little more
                                                (512, 8, 64, 4352, 1024, True),      # 64 rows per expert above hidden 4096
                                                (512, 8, 63, 4352, 1024, False),
                                                (512, 8, 126, 1024, 512, True),      # 126 MB of weights, what the L2 holds
                                                (512, 8, 125, 1024, 512, False), (512, 1, 1024, 7168, 2048, True)])
def test_padding_left_out_and_row_partials_of_the_bf16_calls(monkeypatch, T, K, E, H, I, partials):
    nat, a = _args(T, K, E, H=H, I=I)
    always = nat.SCRATCH_DISPATCHED | nat.SCRATCH_ACTIVATIONS | nat.SCRATCH_GRADIENTS
    used = lambda: nat.lib().mok_layer_scratch(nat.ctypes.byref(a), 0)  # noqa: E731
    assert used() == always | (nat.SCRATCH_ROW_PARTIALS if partials else 0)
    monkeypatch.setenv("MOK_NO_ROW_TRIM", "1")
    assert used() == always
    monkeypatch.setenv("MOK_NO_ROW_TRIM", "0")
    assert used() == always | nat.SCRATCH_ROW_PARTIALS


@pytest.mark.gpu
@pytest.mark.parametrize("E,partials", [(4, False), (16, True)])
def test_memory_beyond_the_outputs(monkeypatch, E, partials):
    import mok
    monkeypatch.setenv("MOK_NO_ROW_TRIM", "0" if partials else "1")
    ops, dev = mok.ops, torch.device("cuda", 0)
    T, H, I, K, MB = 512, 1024, 1024, 2, 16384
    g = torch.Generator(device=dev).manual_seed(8)
    bf = dict(device=dev, dtype=torch.bfloat16)
    normal = lambda *s: torch.randn(*s, generator=g, **bf)  # noqa: E731
    x, dy, rw = normal(T, H), normal(T, H), torch.rand(T, K, generator=g, device=dev) + 0.1
    routes = torch.topk(torch.randn(T, E, generator=g, device=dev), K).indices.to(torch.int32)
    sched = ops.schedule(routes[None], E, 8192, 0)
    shared = [normal(I, H) * 0.05, normal(I, H) * 0.05, normal(H, I) * 0.05]
    routed = [normal(E, I, H) * 0.05, normal(E, I, H) * 0.05, normal(E, H, I) * 0.05]
    q = mok.quantize_routed_weights(*routed)
    slots, d_slots, d_rw = torch.zeros(T * K, H, **bf), torch.zeros(T * K, H, **bf), torch.zeros_like(rw)
    p = lambda t: (t, [t.data_ptr()])  # noqa: E731
    tail = (K, None, 40, MB, 256, None, None, None, None)
    bufs = (*p(dy), *p(d_slots), *p(rw), *p(d_rw))

    def measured(op, *args):
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        out = op(*args)
        taken = torch.cuda.max_memory_allocated() - before
        torch.cuda.synchronize()
        ops.check_status(dev)
        return out, taken - sum(t.untyped_storage().nbytes() for t in out)

    e4m3 = lambda n: MB * n * 33 // 32  # noqa: E731  (bytes and scales)
    slack = 1 << 20                     # rounding of the allocator's blocks; an [MB, H] bf16 buffer has 32 MB, the row sums 0.5 MB
    small = 4 * (2 * MB + E)
    fwd, extra = measured(ops.dispatch_mlp_swiglu_combine_fwd_bf16, *p(x), *p(slots), shared[0], routed[0], shared[1], routed[1],
                          shared[2], routed[2], *sched, *tail, True)
    assert extra <= slack
    _, extra = measured(ops.dispatch_mlp_swiglu_combine_bwd_bf16, *bufs, shared[0], routed[0], shared[1], routed[1], shared[2],
                        routed[2], *fwd[:7], *p(x), *sched, *tail, True)
    sums = MB * (I // 128) * 4 if partials else 0
    assert sums <= extra <= small + sums + (1 << 17)
    fwd, extra = measured(ops.dispatch_mlp_swiglu_combine_fwd_mxfp8, *p(x), *p(slots), shared[0], q[0][0], q[0][1], shared[1], q[1][0],
                          q[1][1], shared[2], q[2][0], q[2][1], *sched, *tail, True)
    assert extra <= e4m3(H) + e4m3(I) + slack
    again, extra = measured(ops.recompute_forward_context_mxfp8, *p(x), shared[0], q[0][0], q[0][1], shared[1], q[1][0], q[1][1],
                            *sched, *tail)
    assert extra <= e4m3(H) + e4m3(I) + slack
    _, extra = measured(ops.dispatch_mlp_swiglu_combine_bwd_mxfp8, *bufs, shared[0], q[0][2], q[0][3], shared[1], q[1][2], q[1][3],
                        shared[2], q[2][2], q[2][3], *again, *p(x), q[0][0], q[0][1], q[1][0], q[1][1], *sched, *tail, True)
    assert extra <= 2 * e4m3(H) + 3 * e4m3(I) + small + MB * (I // 128) * 4 + slack
