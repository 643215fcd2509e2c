"""Mask search and dual compression on both sides of the block counts at which the kernel's form with fewer resident CTAs gives way:
bit for bit against the oracle, single matrices and lists."""
import pytest
import torch

from oracle import sp24_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _check(w, mask, wm, p, pt):
    assert torch.equal(mask.cpu(), wm)
    for (packed, meta), (d, dm) in ((p, (w, wm)), (pt, (w.t().contiguous(), wm.t().contiguous()))):
        a, b = O.compress_with_mask(d, dm, packed.dtype)
        assert torch.equal(packed.cpu().contiguous().view(torch.int16), a.view(torch.int16)) and torch.equal(meta.cpu(), b)


# blocks of 64 x 128 per SM: the lines of the float32 search, the 16-bit search, the 16-bit form with given masks, the list's search
@pytest.mark.parametrize("dtype,lines", [(torch.float32, (2,)), (torch.float16, (3, 4, 13)), (torch.bfloat16, (3,))])
@pytest.mark.parametrize("past", [False, True])
@pytest.mark.parametrize("k", [128, 384])
def test_forms_agree_with_the_oracle(dtype, lines, past, k):
    import sparse
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for line in lines:
        blocks = line * sms // (k // 128) // 2 * 2 + (2 if past else 0)          # rows in steps of 128
        g = torch.Generator().manual_seed(line + k)
        w = (torch.randn(64 * blocks, k, generator=g) * 0.02).to(dtype)
        wm = O.transposable_mask(w)
        wd = w.to(DEV)
        for given in (None, wm.to(DEV)):
            mask, p, pt = sparse.select_and_compress(wd, mask=given)
            _check(w, mask, wm, p, pt)
        for reselect in (True, False):
            masks = [wm.to(DEV) if not reselect else torch.ones(64 * blocks, k, dtype=torch.bool, device=DEV)]
            mask, p, pt = sparse.select_and_compress_many([wd], masks, reselect=reselect)[0]
            _check(w, mask, wm, p, pt)
