"""CPU check of the CTA-pair GEMM's tile rule: only widths that the instruction takes, and which of them are reached."""
import random

import pytest

import _pair_tiles as P


@pytest.mark.parametrize("form", [P.PLAIN, P.FUSED, P.FLOAT8])
def test_rule_takes_legal_widths_only(form):
    from sparse import _ext
    rng = random.Random(form)
    rule = _ext.lib().sp24_pair_tile_columns
    for sms in (2, 80, 132, 148, 160):
        for _ in range(2000):
            ms, n = 256 * rng.randint(1, 64), int(2 ** rng.uniform(0, 22))
            assert rule(ms, n, form, sms) in P.WIDTHS[form], (ms, n, sms)
    assert set(P.shapes(form)) == P.WIDTHS[form]          # every width is reached, so the GPU tests' shapes cover them all
    assert rule(128, 64, form, 148) == 0 and rule(256, 0, form, 148) == 0


@pytest.mark.parametrize("code,says", [(3, "wait gave up (role code 3)"), (11, "1024-byte boundary")])
def test_status_codes_say_what_happened(monkeypatch, code, says):
    """A kernel that could not start is not reported as a wait that gave up; the word is cleared once it was reported."""
    from types import SimpleNamespace

    import torch
    from sparse import spmm
    word = torch.tensor([code], dtype=torch.int32)
    monkeypatch.setattr(spmm, "_ext", SimpleNamespace(host=SimpleNamespace(status_words=lambda: {0: word})))
    with pytest.raises(RuntimeError) as e:
        spmm.check_status()
    assert says in str(e.value) and ("wait" in str(e.value)) == (code != 11) and "cuda:0" in str(e.value)
    spmm.check_status()


def test_slices_of_k_fit_every_floor_plan():
    """The number of slices, which decides the order of the sums, follows from sizes and the number of SMs alone, and its clusters all fit
    at once whichever way the SMs (an even number in each of eight GPCs) are spread."""
    from sparse import _ext
    rule, rng = _ext.lib().sp24_k_slices, random.Random(1)
    edges = [(13, 4), (14, 3), (20, 3), (21, 2), (33, 2), (34, 1)]
    assert [rule(256 * t, 1, 1024, 148) for t, _ in edges] == [s for _, s in edges]
    assert rule(13 * 256 + 128, 63, 960, 148) == 3 and rule(512, 64, 4096, 148) == 1 and rule(512, 1, 896, 148) == 1
    assert rule(100, 1, 1024, 148) == 0 and rule(256, 0, 1024, 148) == 0
    for _ in range(3000):
        sms, plan = rng.choice([132, 144, 148, 152, 160]), [0] * 8
        for _ in range(sms // 2):
            plan[min(rng.randrange(8), rng.randrange(8))] += 2
        tiles = rng.randint(1, 40)
        s = rule(256 * tiles, rng.randint(1, 63), 128 * rng.randint(8, 40), sms)
        assert s == 1 or tiles <= sum(gpc // (2 * s) for gpc in plan)
