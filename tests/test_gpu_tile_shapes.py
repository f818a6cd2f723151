"""Tile shapes of the tcgen05 contraction (tile width, orientation, 64-row tiles, half stages): the shape
the launcher picks gives the same bits as the 128 x 256 tile, at the edges of tiles and ranges."""
import numpy as np
import pytest

from test_gpu_contract import split

pytestmark = pytest.mark.gpu

# (M, N, K): few rows with long and short K, rows that fill 64 / 128 / 192 / 256-wide tiles with and
# without remainders, one row, one column, many tiles
SHAPES = [(1, 1, 64), (3, 45, 3072), (3, 1035, 1088), (65, 17, 64), (96, 1000, 128), (129, 257, 320), (192, 2500, 192),
          (192, 64, 2048), (240, 130, 640), (257, 4999, 128), (1536, 136, 512), (20000, 96, 64)]


@pytest.mark.parametrize("mode", ["bf16", "bf16x3", "tf32x3"])
@pytest.mark.parametrize("shape", SHAPES)
def test_chosen_tile_shape_is_bit_identical(cuda, mode, shape, monkeypatch):
    torch = cuda
    from tdscha_b200 import _native
    M, N, K = shape
    g = torch.Generator(device="cpu").manual_seed(M + 5 * N + K)
    A = torch.randn(M, K, generator=g, dtype=torch.float64).cuda()
    B = torch.randn(N, K, generator=g, dtype=torch.float64).cuda()
    ah, al, ahd, ald = split(torch, A, mode)
    bh, bl, bhd, bld = split(torch, B, mode)
    three = mode.endswith("x3")
    out = {}
    for tile in ("256", None):
        if tile:
            monkeypatch.setenv("TDSCHA_TILE_N", tile)
        else:
            monkeypatch.delenv("TDSCHA_TILE_N")
        D = torch.full((M + 1, N + 3), float("nan"), dtype=torch.float32, device="cuda")
        _native.tc_contract(mode, ah, al if three else None, bh, bl if three else None, D)
        torch.cuda.synchronize()
        assert torch.isnan(D[M]).all() and torch.isnan(D[:, N:]).all()   # nothing written outside M x N
        out[tile] = D[:M, :N].clone()
    assert torch.equal(out[None], out["256"])
    ref = ahd @ bhd.T
    if three:
        ref = ref + ahd @ bld.T + ald @ bhd.T
    err = ((out[None].double() - ref).abs() / (ahd.abs() @ bhd.abs().T)).max().item()
    # fp32 tensor-core accumulation of K products relative to sum |a||b| (the bound of test_gpu_contract)
    assert err < (4e-7 if mode.startswith("bf16") else 1.2e-6) * np.sqrt(K / 64) + 2e-7
