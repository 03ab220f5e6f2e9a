"""Rows-form tile order in groups of m tiles (taken when one expert's weights outgrow L2): the tile list on the CPU with
the kernels' own `decode_tile`, one GEMM of that size on the GPU, and every other rows form of the layer and the router with
the width forced."""
import os
import shutil
import subprocess

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_grouped_tile_list_covers_every_tile_once(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc to build the host harness")
    exe = str(tmp_path / "rows_group_host")
    build = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-O1",
                            "-o", exe, os.path.join(ROOT, "tests", "rows_group_host.cu")], capture_output=True, text=True, timeout=600)
    assert build.returncode == 0, build.stderr[-3000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.startswith("ok"), run.stdout[-2000:] + run.stderr[-2000:]


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [[2304], [1280, 0, 2816]])   # 9 m tiles; groups that span two experts, 16 in all
def test_large_weight_gemm_matches_fp32(counts):
    from mok import _native as nat
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(3)
    rows, N, K, E = sum(counts), 4096, 8704, len(counts)      # 71 MB of weights per expert
    A = torch.randn(rows, K, generator=g, device=dev, dtype=torch.bfloat16)
    B = torch.randn(E, N, K, generator=g, device=dev, dtype=torch.bfloat16) * 0.1
    D = torch.full((rows, N), float("nan"), device=dev, dtype=torch.bfloat16)
    tpe = torch.tensor(counts, dtype=torch.int32, device=dev)
    nt = torch.tensor([rows], dtype=torch.int32, device=dev)
    nat.check(nat.lib().mok_grouped_gemm_bf16(nat.ptr(A), nat.ptr(B), nat.ptr(D), nat.ptr(tpe), nat.ptr(nt), E, rows, N, K, 0,
                                              nat.ptr(nat.status_word(dev)), nat.stream_ptr(dev)), "grouped_gemm")
    nat.check_status(dev)
    off = 0
    for e, n in enumerate(counts):
        ref = A[off:off + n].float() @ B[e].float().T
        # one bf16 rounding of an fp32 sum: at most 2^-9 per element
        assert n == 0 or (D[off:off + n].float() - ref).norm() <= 2.0 ** -9 * ref.norm()
        off += n


def _fixed_capacity(sched, rows_per_expert, length):
    """The schedule with every expert padded to `rows_per_expert` rows: whole tiles of padding, which the routed form skips."""
    peer, token, _, counts = sched
    E, first = counts.numel(), 0
    out_peer, out_token = torch.full((length,), -1, dtype=torch.int32, device=peer.device), torch.zeros(length, dtype=torch.int32, device=peer.device)
    for e, n in enumerate(int(c) for c in counts):
        assert n <= rows_per_expert
        out_peer[e * rows_per_expert:e * rows_per_expert + n] = peer[first:first + n]
        out_token[e * rows_per_expert:e * rows_per_expert + n] = token[first:first + n]
        first += n
    return (out_peer, out_token, torch.full((1,), E * rows_per_expert, dtype=torch.int32, device=peer.device),
            torch.full_like(counts, rows_per_expert))


@pytest.mark.gpu
@pytest.mark.parametrize("mxfp8", [False, True])
@pytest.mark.parametrize("skip", [False, True])                      # rows kept, or stored into the slots by the epilogue
@pytest.mark.parametrize("T,K,E,pad,MB,no_trim", [(1536, 2, 5, 0, 8192, "1"), (1536, 2, 5, 0, 2560, "1"), (768, 2, 21, 0, 8192, "0"),
                                                  (768, 2, 13, 512, 8192, "0")])
def test_layer_is_the_same_for_every_group_width(monkeypatch, mxfp8, skip, T, K, E, pad, MB, no_trim):
    """Fused, dual, scattered, routed and MXFP8 rows forms: bitwise what m tile major order gives, with ragged experts, several
    windows, a last group that is narrower than the others and tiles that hold padding only."""
    import mok
    ops, dev, H, I = mok.ops, torch.device("cuda", 0), 512, 768
    g = torch.Generator(device=dev).manual_seed(12)
    bf = dict(device=dev, dtype=torch.bfloat16)
    normal = lambda *s: torch.randn(*s, generator=g, **bf)  # noqa: E731
    x, dy, rw = normal(T, H), normal(T, H), torch.rand(T, K, generator=g, device=dev) + 0.1
    skew = torch.linspace(-1.0, 0.4, E, device=dev)
    routes = torch.topk(torch.randn(T, E, generator=g, device=dev) + skew, K).indices.to(torch.int32)
    sched = ops.schedule(routes[None], E, 8192, 0)
    if pad:
        sched = _fixed_capacity(sched, pad, 8192)
    m_tiles = min(int(sched[2]), MB) // 256
    assert m_tiles > 8 and m_tiles % 8 != 0
    shared = [normal(I, H) * 0.05, normal(I, H) * 0.05, normal(H, I) * 0.05]
    routed = [normal(E, I, H) * 0.05, normal(E, I, H) * 0.05, normal(E, H, I) * 0.05]
    q = mok.quantize_routed_weights(*routed) if mxfp8 else None
    tail = (K, None, 40, MB, 256, None, None, None, None, skip)
    p = lambda t: (t, [t.data_ptr()])  # noqa: E731

    def run():
        slots, d_slots, d_rw = torch.zeros(T * K, H, **bf), torch.zeros(T * K, H, **bf), torch.zeros_like(rw)
        bufs = (*p(dy), *p(d_slots), *p(rw), *p(d_rw))
        if mxfp8:
            fwd = ops.dispatch_mlp_swiglu_combine_fwd_mxfp8(
                *p(x), *p(slots), shared[0], q[0][0], q[0][1], shared[1], q[1][0], q[1][1], shared[2], q[2][0], q[2][1], *sched, *tail)
            bwd = ops.dispatch_mlp_swiglu_combine_bwd_mxfp8(
                *bufs, shared[0], q[0][2], q[0][3], shared[1], q[1][2], q[1][3], shared[2], q[2][2], q[2][3], *fwd[:11], *p(x),
                q[0][0], q[0][1], q[1][0], q[1][1], *sched, *tail)
            grads = bwd[12:]
        else:
            fwd = ops.dispatch_mlp_swiglu_combine_fwd_bf16(*p(x), *p(slots), shared[0], routed[0], shared[1], routed[1], shared[2],
                                                           routed[2], *sched, *tail)
            bwd = ops.dispatch_mlp_swiglu_combine_bwd_bf16(*bufs, shared[0], routed[0], shared[1], routed[1], shared[2], routed[2],
                                                           *fwd[:7], *p(x), *sched, *tail)
            grads = bwd[9:]
        torch.cuda.synchronize()
        ops.check_status(dev)
        return [slots, d_slots, d_rw, *grads]

    monkeypatch.setenv("MOK_NO_ROW_TRIM", no_trim)
    monkeypatch.setenv("MOK_ROWS_GROUP", "1")
    want = run()
    for width in ("4", "8"):
        monkeypatch.setenv("MOK_ROWS_GROUP", width)
        for i, (a, b) in enumerate(zip(want, run())):
            assert a.float().abs().sum() > 0 and torch.equal(a, b), (width, i)


@pytest.mark.gpu
def test_router_logits_are_the_same_for_every_group_width(monkeypatch):
    import mok
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(13)
    x, w = torch.randn(2816, 512, generator=g, device=dev, dtype=torch.bfloat16), torch.randn(300, 512, generator=g, device=dev)
    monkeypatch.setenv("MOK_ROWS_GROUP", "1")                         # 11 m tiles, 2 column tiles, two terms of the weight
    want = mok.ops.router_fwd(x, w, None, 8)
    monkeypatch.setenv("MOK_ROWS_GROUP", "8")
    for a, b in zip(want, mok.ops.router_fwd(x, w, None, 8)):
        assert torch.equal(a, b)
    mok.ops.check_status(dev)
