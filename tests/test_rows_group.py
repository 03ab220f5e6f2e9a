"""Rows-form tile order in groups of m tiles (taken when one expert's weights outgrow L2): the tile list on the CPU with
the kernels' own `decode_tile`, and one GEMM of that size on the GPU."""
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
