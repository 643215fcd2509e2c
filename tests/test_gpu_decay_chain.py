"""Masked decays in a row, each reading what the one before has just written (their inputs are asked for before the wait): sizes around a
block's 4096 elements, every mask type, unaligned masks.  Exact: a product and a sum, each rounded once."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("mask_dtype", [torch.bool, torch.float16, torch.float32])
@pytest.mark.parametrize("n", [3, 4, 33, 4095, 4096, 4101, 148 * 4096 + 36, 3 << 20])
def test_decays_in_a_row(n, mask_dtype):
    import sparse
    g = torch.Generator(device=DEV).manual_seed(n)
    a, b = (torch.randn(n, device=DEV, generator=g) for _ in range(2))
    keep = torch.zeros(n + 4, device=DEV, dtype=mask_dtype)[4:]      # 4 elements off the buffer's start
    keep.copy_(torch.rand(n, device=DEV, generator=g) < 0.5)
    ra, rb = a.clone(), b.clone()
    torch.cuda.synchronize()
    for i in range(6):
        sparse.masked_add_(a, b, keep, alpha=0.5 + i)
        sparse.masked_add_(b, a, keep, alpha=-0.25)
    for i in range(6):
        ra = torch.where(keep != 0, ra, ra + rb * (0.5 + i))
        rb = torch.where(keep != 0, rb, rb + ra * -0.25)
    assert torch.equal(a, ra) and torch.equal(b, rb)


@pytest.mark.parametrize("mask_dtype", [torch.bool, torch.float32])
@pytest.mark.parametrize("blocks", [296, 297, 740, 741, 2100, 2800])
def test_decays_whose_blocks_ask_ahead_or_not(blocks, mask_dtype):
    """Either side of two and of five blocks an SM, and of what L2 holds of the three arrays (float32 masks: from 2049 blocks, bool from 2731)."""
    test_decays_in_a_row(blocks * 4096 - 2048 + 7, mask_dtype)
