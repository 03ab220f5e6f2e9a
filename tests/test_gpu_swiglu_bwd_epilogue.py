"""SwiGLU backward in the epilogue of the down projection's input gradient (experts of at most 128 rows) against the separate
kernel, which runs when the padding rows are computed too: same d_hidden, d_gate,
d_up and weight gradients bitwise (routed and shared expert, ragged loads, windows with replay), router-weight gradients up
to the order of an fp32 sum of `intermediate` terms."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [None, 0.5])
@pytest.mark.parametrize("T,H,I,E,K,MB", [(512, 256, 256, 8, 1, 512), (768, 512, 768, 24, 4, 2048), (512, 1024, 1280, 16, 2, 8192)])
def test_fused_swiglu_backward_equals_the_separate_kernel(monkeypatch, T, H, I, E, K, MB, limit):
    import mok
    ops, dev = mok.ops, torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(5)
    bf = dict(device=dev, dtype=torch.bfloat16)
    normal = lambda *s: torch.randn(*s, generator=g, **bf)  # noqa: E731
    x, dy, rw = normal(T, H), normal(T, H), torch.rand(T, K, generator=g, device=dev) + 0.1
    routes = torch.topk(torch.randn(T, E, generator=g, device=dev), K).indices.to(torch.int32)
    cap = -(-(2 * T * K + 256 * E) // 512) * 512
    sched = ops.schedule(routes[None], E, cap, 0)
    shared = [normal(I, H) * 0.05, normal(I, H) * 0.05, normal(H, I) * 0.05]
    routed = [normal(E, I, H) * 0.05, normal(E, I, H) * 0.05, normal(E, H, I) * 0.05]

    def run(skip):
        slots, d_slots, d_rw = torch.zeros(T * K, H, **bf), torch.zeros(T * K, H, **bf), torch.zeros_like(rw)
        p = lambda t: (t, [t.data_ptr()])  # noqa: E731
        tail = (K, limit, 40, MB, 256, None, None, None, None, skip)
        fwd = ops.dispatch_mlp_swiglu_combine_fwd_bf16(*p(x), *p(slots), shared[0], routed[0], shared[1], routed[1], shared[2],
                                                       routed[2], *sched, *tail)
        bwd = ops.dispatch_mlp_swiglu_combine_bwd_bf16(
            *p(dy), *p(d_slots), *p(rw), *p(d_rw), shared[0], routed[0], shared[1], routed[1], shared[2], routed[2], *fwd[:7], *p(x),
            *sched, *tail)
        torch.cuda.synchronize()
        ops.check_status(dev)
        return fwd, bwd, d_slots, d_rw

    monkeypatch.setenv("MOK_NO_ROW_TRIM", "1")
    fwd, bwd, d_slots, d_rw = run(False)
    _, _, d_slots_skip, d_rw_skip = run(True)
    assert torch.equal(d_slots, d_slots_skip) and torch.equal(d_rw, d_rw_skip)
    monkeypatch.delenv("MOK_NO_ROW_TRIM")
    rows = int(sched[2])
    n = rows - MB * ((rows - 1) // MB)                           # rows of the last window: what the buffers hold at the end
    # two orders of a sum of I fp32 terms differ by at most 2 I 2^-24 times the sum of the terms' magnitudes
    terms = fwd[6].float().abs().amax() * bwd[7][:n].float().abs().amax() * I
    bound = 2 * I * 2.0 ** -24 * terms / rw.min()
    for skip in (False, True):
        _, b2, ds2, drw2 = run(skip)
        for i, (a, b) in enumerate(zip(bwd, b2)):
            if i in (1, 8):
                continue                                         # not kept, or a buffer this step does not touch
            if i in (3, 5, 7):
                a, b = a[:n], b[:n]
            assert a.float().abs().sum() > 0 and torch.equal(a, b), i
        assert torch.equal(d_slots, ds2)
        assert (d_rw - drw2).abs().max() <= bound and d_rw.abs().sum() > 0
