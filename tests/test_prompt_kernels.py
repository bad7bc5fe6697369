"""Kernels of prompt steps at the edges of their tiles, against plain PyTorch in 64 bits."""
import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from airframe_b200 import kernels
    return kernels


@pytest.mark.parametrize("N, Kd", [(200, 72), (384, 320), (2304, 1032)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_gemm_tensor_cores_token_tiles(K, N, Kd, out_dtype):
    """Every width of a token tile, on one SM with one accumulator or two and on a pair: the same bits, whatever the tile, as
    the chosen one, and the product in 64 bits within the roundings of its output."""
    gen = torch.Generator().manual_seed(N)
    w = (torch.randn(N, Kd, generator=gen) * 0.05).to(DEV, torch.bfloat16)
    for M in (65, 257, 700):
        x = torch.randn(M, Kd, generator=gen).to(DEV, torch.bfloat16)
        want = x.double() @ w.double().T
        first = torch.full((M, N), float("nan"), device=DEV, dtype=out_dtype)
        K.gemm_tc(first, x, w)
        assert ((first.double() - want).abs() <= (2e-6 if out_dtype == torch.float32 else 2.0 ** -8) * want.abs() + 2e-5).all()
        for n_acc in (1, 2, 4):
            for tile in range(32, 257, 32 if n_acc == 4 else 16):
                out = torch.full((M, N), float("nan"), device=DEV, dtype=out_dtype)
                K.gemm_tc(out, x, w, n_acc=n_acc, token_tile=tile)
                assert torch.equal(out, first), (M, n_acc, tile)
