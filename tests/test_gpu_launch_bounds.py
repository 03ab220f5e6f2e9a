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
