"""One rank: where the kernels read an input from (`functional._source`), with a stand-in for the workspace.  Under every
kind of tracing the address must be the staging buffer's: a caller's address would be a constant of the recorded graph."""
import types

import pytest
import torch


def _setup():
    from mok import functional as F
    bufs = {n: torch.zeros(4, 8) for n in ("combine_buffer", "d_x_routed_buffer", "d_router_weight_buffer")}
    ws, stage, seen = types.SimpleNamespace(ep_size=1, **bufs), torch.zeros(4, 8), []

    def f(x):
        source, pointers = F._source(ws, stage, [stage.data_ptr()], x)
        seen.append((source is stage, pointers))
        return source * 2
    return ws, stage, seen, f


def test_eager_calls_read_in_place():
    ws, stage, seen, f = _setup()
    x = torch.randn(4, 8)
    assert torch.equal(f(x), x * 2) and seen == [(False, [x.data_ptr()])]
    f(ws.combine_buffer)
    assert seen[1] == (True, [stage.data_ptr()])


@pytest.mark.parametrize("how", ["make_fx", "make_fx pre_dispatch", "jit.trace"])
def test_traced_calls_are_staged(how):
    from torch.fx.experimental.proxy_tensor import make_fx
    _, stage, seen, f = _setup()
    x, y = torch.randn(4, 8), torch.randn(4, 8)
    if how == "jit.trace":
        graph = torch.jit.trace(f, (x,), check_trace=False)
    else:
        graph = make_fx(f, pre_dispatch="pre" in how)(x)
    assert seen == [(True, [stage.data_ptr()])]
    assert torch.equal(graph(y), y * 2) and torch.equal(stage, y)


@pytest.mark.parametrize("transform", ["vmap", "grad", "functionalize"])
def test_functorch_transforms_are_refused_by_the_copy(transform):
    _, stage, seen, f = _setup()
    call = {"vmap": lambda: torch.func.vmap(f)(torch.randn(2, 4, 8)),
            "grad": lambda: torch.func.grad(lambda x: f(x).sum())(torch.randn(4, 8)),
            "functionalize": lambda: torch.func.functionalize(f)(torch.randn(4, 8))}[transform]
    with pytest.raises(RuntimeError, match="inplace|in-place|mutating"):
        call()
