"""One rank, MXFP8: the quantizer reads the rows' tokens itself; several ranks: a dispatch pass writes the rows first.  The
same schedule reaches both: with a second rank whose tokens all go to its own experts, rank 0 serves exactly what it serves
alone.  Everything the ops return and write has to be bitwise the same (row tiles with padding, several windows, ragged and
empty experts)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skip", [False, True])
@pytest.mark.parametrize("T,H,I,E,K,MB", [(512, 256, 256, 3, 1, 512), (768, 512, 256, 6, 4, 2048), (512, 768, 512, 5, 2, 8192)])
def test_quantizer_that_gathers_equals_dispatch_and_quantize(T, H, I, E, K, MB, skip):
    import mok
    ops, dev = mok.ops, torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(3)
    bf = dict(device=dev, dtype=torch.bfloat16)
    normal = lambda *s: torch.randn(*s, generator=g, **bf)  # noqa: E731
    x, dy, rw = normal(T, H), normal(T, H), torch.rand(T, K, generator=g, device=dev) + 0.1
    scores = torch.randn(T, E, generator=g, device=dev)
    scores[:, E - 1] -= 20.0                                     # (nearly) empty expert
    mine = torch.topk(scores, K).indices.to(torch.int32)
    cap = -(-(2 * T * K + 256 * E) // 512) * 512
    shared = [normal(I, H) * 0.05, normal(I, H) * 0.05, normal(H, I) * 0.05]
    q = mok.quantize_routed_weights(normal(E, I, H) * 0.05, normal(E, I, H) * 0.05, normal(E, H, I) * 0.05)
    tail = (K, None, 40, MB, 256, None, None, None, None, skip)

    def run(ep):
        zeros = lambda: torch.zeros(T * K, H, **bf)  # noqa: E731
        other = [torch.zeros_like(x), torch.zeros_like(dy), torch.ones_like(rw), zeros(), zeros(), torch.zeros_like(rw)]
        slots, d_slots, d_rw = zeros(), zeros(), torch.zeros_like(rw)
        ptrs = lambda a, b: [a.data_ptr(), b.data_ptr()][:ep]  # noqa: E731
        sched = ops.schedule(torch.stack([mine, torch.full_like(mine, E)][:ep]), E, cap, 0)
        xp = ptrs(x, other[0])
        fwd = ops.dispatch_mlp_swiglu_combine_fwd_mxfp8(
            x, xp, slots, ptrs(slots, other[3]), shared[0], q[0][0], q[0][1], shared[1], q[1][0], q[1][1], shared[2], q[2][0],
            q[2][1], *sched, *tail)
        again = ops.recompute_forward_context_mxfp8(x, xp, shared[0], q[0][0], q[0][1], shared[1], q[1][0], q[1][1], *sched, *tail[:-1])
        n = min(int(sched[2]), MB)                               # rows of the first window that carry data
        context = [t.view(torch.uint8).clone() for t in (fwd[0][:, :n], fwd[3][:n], again[0][:, :n], again[9][:, :n])]
        bwd = ops.dispatch_mlp_swiglu_combine_bwd_mxfp8(
            dy, ptrs(dy, other[1]), d_slots, ptrs(d_slots, other[4]), rw, ptrs(rw, other[2]), d_rw, ptrs(d_rw, other[5]),
            shared[0], q[0][2], q[0][3], shared[1], q[1][2], q[1][3], shared[2], q[2][2], q[2][3], *again,
            x, xp, q[0][0], q[0][1], q[1][0], q[1][1], *sched, *tail)
        torch.cuda.synchronize()
        ops.check_status(dev)
        return context + [slots, d_slots, d_rw, *bwd[12:]]

    for i, (a, b) in enumerate(zip(run(1), run(2))):
        assert torch.equal(a, b), i
        assert a.float().abs().sum() > 0, i
