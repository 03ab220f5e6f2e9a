"""GEMM epilogues that store routed rows straight into the token owners' slots, against the same op with a row buffer and
a combine pass: bitwise equal slots and gradients, both precisions.  Two ranks' buffers on one GPU stand in for peers (the
kernels only dereference the addresses they are given); the ring has several windows, experts have ragged loads."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mxfp8", [False, True])
@pytest.mark.parametrize("T,H,I,E,K", [(512, 256, 256, 2, 1), (768, 512, 256, 6, 4)])
def test_scattered_rows_equal_the_combine_pass(mxfp8, T, H, I, E, K):
    import mok
    ops, dev, ep = mok.ops, torch.device("cuda", 0), 2
    g = torch.Generator(device=dev).manual_seed(9)
    bf = dict(device=dev, dtype=torch.bfloat16)
    normal = lambda *s: torch.randn(*s, generator=g, **bf)  # noqa: E731
    xs, dys = [normal(T, H) for _ in range(ep)], [normal(T, H) for _ in range(ep)]
    rws = [torch.rand(T, K, generator=g, device=dev) + 0.1 for _ in range(ep)]
    topk_all = torch.stack([torch.topk(torch.randn(T, 2 * E, generator=g, device=dev), K).indices for _ in range(ep)]).to(torch.int32)
    cap = -(-(ep * T * K + 256 * E) // 512) * 512
    sched = ops.schedule(topk_all, E, cap, 0)
    shared = [normal(I, H) * 0.05, normal(I, H) * 0.05, normal(H, I) * 0.05]
    routed = [normal(E, I, H) * 0.05, normal(E, I, H) * 0.05, normal(E, H, I) * 0.05]
    q = mok.quantize_routed_weights(*routed)
    addr = lambda ts: [t.data_ptr() for t in ts]  # noqa: E731
    tail = (K, None, 40, 1024, 256, None, None, None, None)

    def run(skip):
        slots = [torch.zeros(T * K, H, **bf) for _ in range(ep)]
        d_slots = [torch.zeros(T * K, H, **bf) for _ in range(ep)]
        d_rws = [torch.zeros(T, K, device=dev) for _ in range(ep)]
        bufs = (dys[0], addr(dys), d_slots[0], addr(d_slots), rws[0], addr(rws), d_rws[0], addr(d_rws))
        if mxfp8:
            fwd = ops.dispatch_mlp_swiglu_combine_fwd_mxfp8(
                xs[0], addr(xs), slots[0], addr(slots), shared[0], q[0][0], q[0][1], shared[1], q[1][0], q[1][1], shared[2],
                q[2][0], q[2][1], *sched, *tail, skip)
            bwd = ops.dispatch_mlp_swiglu_combine_bwd_mxfp8(
                *bufs, shared[0], q[0][2], q[0][3], shared[1], q[1][2], q[1][3], shared[2], q[2][2], q[2][3], *fwd[:11],
                xs[0], addr(xs), q[0][0], q[0][1], q[1][0], q[1][1], *sched, *tail, skip)
            grads = bwd[12:]
        else:
            fwd = ops.dispatch_mlp_swiglu_combine_fwd_bf16(
                xs[0], addr(xs), slots[0], addr(slots), shared[0], routed[0], shared[1], routed[1], shared[2], routed[2],
                *sched, *tail, skip)
            bwd = ops.dispatch_mlp_swiglu_combine_bwd_bf16(
                *bufs, shared[0], routed[0], shared[1], routed[1], shared[2], routed[2], *fwd[:7], xs[0], addr(xs),
                *sched, *tail, skip)
            grads = bwd[9:]
        assert fwd[-1].shape[0] == bwd[1].shape[0] == (0 if skip else 1024)
        torch.cuda.synchronize()
        ops.check_status(dev)
        return slots + d_slots + d_rws + list(grads)

    for i, (a, b) in enumerate(zip(run(False), run(True))):
        assert a.float().abs().sum() > 0 and torch.equal(a, b), i
