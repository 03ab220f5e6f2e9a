"""Rows GEMMs with the tokens on the N side of the MMA (padding rows left out) against the GEMMs that run over the padding:
every output bitwise equal, padding rows zero in both.  Both forms are forced.  Loads of 0, 1, 63, 64, 65, 128, 129, 255, 256,
257 ... rows give every width of the last tile; several windows; slots written by the GEMM or by a combine pass; with and without
the clamp."""
import pytest
import torch

pytestmark = pytest.mark.gpu
LOADS = [0, 1, 63, 64, 65, 128, 129, 191, 192, 193, 255, 256, 257, 511, 2, 7, 31, 32, 33, 0, 40, 16, 320, 0]


@pytest.mark.parametrize("H,I,MB,limit", [(256, 256, 8192, None), (768, 512, 2048, 0.5), (1280, 1024, 512, None)])
@pytest.mark.parametrize("skip", [False, True])
def test_padding_left_out_changes_nothing(monkeypatch, H, I, MB, limit, skip):
    import mok
    ops, dev = mok.ops, torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(11)
    bf = dict(device=dev, dtype=torch.bfloat16)
    normal = lambda *s: torch.randn(*s, generator=g, **bf)  # noqa: E731
    E = len(LOADS)
    routes = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(LOADS)])
    T = -(-routes.numel() // 256) * 256
    routes = torch.cat([routes, torch.full((T - routes.numel(),), E - 2, dtype=torch.int32)])
    routes = routes[torch.randperm(T, generator=torch.Generator().manual_seed(2))].to(dev)[:, None].contiguous()
    x, dy, rw = normal(T, H), normal(T, H), torch.rand(T, 1, generator=g, device=dev) + 0.1
    sched = ops.schedule(routes[None], E, T + 256 * E, 0)
    shared = [normal(I, H) * 0.05, normal(I, H) * 0.05, normal(H, I) * 0.05]
    routed = [normal(E, I, H) * 0.05, normal(E, I, H) * 0.05, normal(E, H, I) * 0.05]
    rows = int(sched[2])
    last = rows - MB * ((rows - 1) // MB)                        # rows that the buffers hold after the last window

    def run():
        slots, d_slots, d_rw = torch.zeros(T, H, **bf), torch.zeros(T, H, **bf), torch.zeros_like(rw)
        p = lambda t: (t, [t.data_ptr()])  # noqa: E731
        tail = (1, limit, 40, MB, 256, None, None, None, None, skip)
        fwd = ops.dispatch_mlp_swiglu_combine_fwd_bf16(*p(x), *p(slots), shared[0], routed[0], shared[1], routed[1], shared[2],
                                                       routed[2], *sched, *tail)
        n = min(rows, MB)
        again = ops.recompute_forward_context_bf16(*p(x), shared[0], routed[0], shared[1], routed[1], *sched, *tail[:-1])
        context = [fwd[i][:n].clone() for i in (0, 2, 4, 6)] + ([] if skip else [fwd[8][:n].clone()])
        context += [again[i][:n].clone() for i in (0, 2, 4, 6)]
        bwd = ops.dispatch_mlp_swiglu_combine_bwd_bf16(
            *p(dy), *p(d_slots), *p(rw), *p(d_rw), shared[0], routed[0], shared[1], routed[1], shared[2], routed[2], *again, *p(x),
            *sched, *tail)
        torch.cuda.synchronize()
        ops.check_status(dev)
        kept = [bwd[i][:last] for i in (3, 5)] + ([] if skip else [bwd[1][:last], bwd[7][:last]])
        return context + kept + [slots, d_slots, *bwd[9:]], d_rw

    monkeypatch.setenv("MOK_NO_ROW_TRIM", "0")
    trimmed, trimmed_rw = run()
    monkeypatch.setenv("MOK_NO_ROW_TRIM", "1")
    padded, padded_rw = run()
    for i, (a, b) in enumerate(zip(padded, trimmed)):
        assert a.float().abs().sum() > 0 and torch.equal(a, b), i
    # sums of I fp32 terms in another order: the gradients are O(1) here, 2 I 2^-24 of the sum of magnitudes bounds them
    assert (padded_rw - trimmed_rw).abs().max() <= 2 * I * 2.0 ** -24 * padded_rw.abs().amax() * I ** 0.5
