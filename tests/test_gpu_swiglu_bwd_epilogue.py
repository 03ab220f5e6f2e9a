"""SwiGLU backward in the epilogue of the down projection's input gradient (taken for experts of few rows, forced here) against the separate
kernel, which runs when the padding rows are computed too: same d_hidden, d_gate, d_up and weight gradients bitwise (routed and
shared expert, ragged loads, windows with replay).  The router-weight gradients of both are sums of `intermediate` fp32 terms in
an order of their own; each is checked, route by route, against the float64 sum of that route's own terms."""
import pytest
import torch


def router_gradient(gate, up, d_hidden, weight, limit):
    """Per row: sum(d_hidden * silu(gate) * up) / weight in float64, how far an fp32 sum of the same terms in any order may be
    from it, and the least of what leaving out one block of 128 columns would change it by."""
    g, u, dh, w = gate.double(), up.double(), d_hidden.double(), weight.double()
    assert g.abs().max() <= 20
    if limit is not None:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    terms = dh * g * torch.sigmoid(g) * u
    # n additions of at most 2^-24 of the magnitudes' sum each, the quotient's and the products' few roundings, and per term
    # the error of __expf, 2 + 1.16 |gate| units in the last place (2^-23), and of the division behind it: below 2^-18 here
    bound = ((g.shape[1] + 8) * 2.0 ** -24 + 2.0 ** -18) * terms.abs().sum(1) / w
    return terms.sum(1) / w, bound, terms.unflatten(1, (-1, 128)).sum(2).abs().amin(1) / w


def test_router_gradient_bound_tells_a_missing_block():
    g = torch.Generator().manual_seed(3)
    for H, I, limit in ((256, 256, None), (512, 768, 0.5), (1024, 1280, None), (1024, 1280, 0.5)):
        gate, up, dh = (torch.randn(512, I, generator=g) * std for std in (0.05 * H ** 0.5, 0.05 * H ** 0.5, 0.05 * H ** 0.5))
        _, bound, block = router_gradient(gate, up, dh, torch.rand(512, generator=g) + 0.1, limit)
        assert (block > 2 * bound).float().mean() > 0.8


@pytest.mark.gpu
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

    def run(skip, MB=MB):
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
    rows = int(sched[2])
    n = rows - MB * ((rows - 1) // MB)                           # rows of the last window: what the buffers hold at the end
    whole = -(-rows // 256) * 256                                # one window: the buffers hold every row's terms
    fwd, bwd_whole, _, _ = run(False, whole)
    used = sched[0][:rows] >= 0
    route = sched[1][:rows][used].long()
    want, bound, block = router_gradient(*(t[:rows][used] for t in (fwd[2], fwd[4], bwd_whole[7])), rw.flatten()[route], limit)
    assert (block > 2 * bound).float().mean() > 0.8              # a missing block of 128 columns would show

    def check_router_gradient(got):
        assert ((got.flatten()[route].double() - want).abs() <= bound).all()

    check_router_gradient(d_rw)
    monkeypatch.setenv("MOK_NO_ROW_TRIM", "0")
    for skip in (False, True):
        _, b2, ds2, drw2 = run(skip)
        for i, (a, b) in enumerate(zip(bwd, b2)):
            if i in (1, 8):
                continue                                         # not kept, or a buffer this step does not touch
            if i in (3, 5, 7):
                a, b = a[:n], b[:n]
            assert a.float().abs().sum() > 0 and torch.equal(a, b), i
        assert torch.equal(d_slots, ds2)
        check_router_gradient(drw2)
