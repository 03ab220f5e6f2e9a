"""The layer's launches cover the rows that the routes can fill, not the schedule's capacity."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu


def _layer(dist_ctx, T, K, E, claim=None):
    import torch.distributed as dist
    import mok
    F = mok.functional
    dev = dist_ctx[2]
    inp = O.make_rank_inputs(0, E, E, K, T, 256, 256)
    d = {k: v.to(dev) for k, v in vars(inp).items()}
    config = F.MoKConfig(minibatch_size=256, macrobatch_size=512, schedule_capacity_multiplier=4.0)
    ws = F.get_workspace(config, dist.group.WORLD, device=dev, num_local_tokens=T, hidden_size=256, topk=K)
    sched = F.build_schedule(ws, config, d["topk_experts"], num_local_experts=E)
    if claim is not None:
        sched.num_tokens.fill_(claim)
    w = [d[n] for n in ("w_shared_gate", "w_shared_up", "w_shared_down", "w_routed_gate", "w_routed_up", "w_routed_down")]
    out, _ = F.forward(config, ws, sched, d["x"], d["router_weights"], *w)
    torch.cuda.synchronize()
    return inp, out


@pytest.mark.parametrize("T,K,E", [(512, 1, 1), (512, 1, 3), (1024, 3, 5), (512, 2, 8)])
def test_every_row_is_covered(dist_ctx, T, K, E):
    import mok
    inp, out = _layer(dist_ctx, T, K, E)
    mok.ops.check_status(dist_ctx[2])
    ref = O.moe_layer_oracle([inp])[0].output.float()
    assert (out.float().cpu() - ref).norm() <= 1e-2 * ref.norm()     # the acceptance bound of the layer


def test_schedule_that_claims_more_rows_is_reported(dist_ctx):
    import mok
    _, out = _layer(dist_ctx, 512, 1, 1, claim=1024)     # one expert, 512 routes: 512 rows
    assert torch.isnan(out.float()).all()
    with pytest.raises(RuntimeError, match="claims more rows"):
        mok.ops.check_status(dist_ctx[2])


@pytest.mark.parametrize("mxfp8", [False, True])
@pytest.mark.parametrize("T,K,E,no_trim", [(1024, 2, 3, "1"), (512, 1, 8, "0")])   # GEMMs over the padding rows, and without them
def test_experts_padded_to_a_fixed_capacity(dist_ctx, monkeypatch, T, K, E, no_trim, mxfp8):
    """A schedule that did not come from `schedule` may pad its experts as it likes: with 1024 rows per expert, nearly all of
    them padding, slots, outputs and gradients are bitwise those of the compact schedule, through the functional calls and
    the ops, in several windows (an expert each, so that no gradient is a sum over windows)."""
    import dataclasses

    import torch.distributed as dist
    import mok
    F, dev, cap_e = mok.functional, dist_ctx[2], 1024
    monkeypatch.setenv("MOK_NO_ROW_TRIM", no_trim)
    inp = O.make_rank_inputs(0, E, E, K, T, 256, 256)
    d = {k: v.to(dev) for k, v in vars(inp).items()}
    routed = [d[n] for n in ("w_routed_gate", "w_routed_up", "w_routed_down")]
    shared = [d[n] for n in ("w_shared_gate", "w_shared_up", "w_shared_down")]
    back = routed
    if mxfp8:
        q = mok.quantize_routed_weights(*routed)
        routed, back = (q[0][:2], q[1][:2], q[2][:2]), (q[0], q[1], q[2][2:])

    def run(padded, macrobatch):
        config = F.MoKConfig(minibatch_size=256, macrobatch_size=macrobatch, schedule_capacity_multiplier=float(cap_e * E // (T * K) + 1))
        ws = F.get_workspace(config, dist.group.WORLD, device=dev, num_local_tokens=T, hidden_size=256, topk=K)
        sched = F.build_schedule(ws, config, d["topk_experts"], num_local_experts=E)
        if padded:
            counts = [int(n) for n in sched.tokens_per_expert]
            assert max(counts) <= cap_e and cap_e * E > sched.max_rows and cap_e * E <= ws.schedule_capacity
            peer, token, first = torch.full_like(sched.peer_rank, -1), torch.zeros_like(sched.peer_token_idx), 0
            for e, n in enumerate(counts):
                peer[e * cap_e:e * cap_e + n] = sched.peer_rank[first:first + n]
                token[e * cap_e:e * cap_e + n] = sched.peer_token_idx[first:first + n]
                first += n
            sched = dataclasses.replace(sched, peer_rank=peer, peer_token_idx=token, num_tokens=torch.full_like(sched.num_tokens, cap_e * E),
                                        tokens_per_expert=torch.full_like(sched.tokens_per_expert, cap_e))
        out, ctx = F.forward(config, ws, sched, d["x"], d["router_weights"], *shared, *routed)
        slots = ws.combine_buffer.clone()
        ctx = F.recompute_forward_context(config, ws, sched, d["x"], *shared[:2], *routed[:2])
        grads = F.backward(config, ws, sched, ctx, d["d_output"], d["x"], d["router_weights"], *shared, *back)
        torch.cuda.synchronize()
        mok.ops.check_status(dev)
        return [out, slots, *grads]

    want = run(False, cap_e * E)
    for i, (a, b) in enumerate(zip(want, run(True, cap_e))):
        assert a.float().abs().sum() > 0 and torch.equal(a, b), i
