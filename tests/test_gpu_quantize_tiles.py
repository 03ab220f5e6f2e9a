"""Quantizer blocks that walk several column tiles: a matrix set large enough for two or eight tiles per block, with column
counts that these do not divide, against calls so small that every block takes one tile.  Bitwise equal, both layouts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts,rows,cols", [(1, 128, 128), (9, 2048, 2432), (18, 4096, 2432), (1, 65536, 2176)])
@pytest.mark.parametrize("normal,transposed", [(True, True), (True, False), (False, True)])
def test_large_quantization_equals_small_calls(experts, rows, cols, normal, transposed):
    import mok
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(1)
    x = torch.randn(experts, rows, cols, generator=g, device=dev, dtype=torch.bfloat16)
    x[:, ::37] *= 1e-3
    x[0, 5, 7], x[0, 0, 1], x[-1, -1, -1] = float("inf"), float("nan"), 1e-39
    whole = mok.ops.mxfp8_quantize(x, normal, transposed)
    as_bytes = lambda t: t.view(torch.uint8)  # noqa: E731
    for e, r0 in ((0, 0), (experts - 1, rows - 128), (experts // 2, (rows // 256) * 128)):
        part = mok.ops.mxfp8_quantize(x[e, r0:r0 + 128].contiguous(), normal, transposed)
        if normal:
            assert torch.equal(as_bytes(whole[0][e, r0:r0 + 128]), as_bytes(part[0]))
            assert torch.equal(whole[1][(e * rows + r0) // 128], part[1][0])
        if transposed:
            assert torch.equal(as_bytes(whole[2][e, :, r0:r0 + 128].contiguous()), as_bytes(part[2]))
            assert torch.equal(whole[3][e * (cols // 128):(e + 1) * (cols // 128), r0 // 128], part[3][:, 0])
