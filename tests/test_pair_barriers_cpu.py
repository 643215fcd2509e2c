"""CPU model of the accumulator barriers of the CTA-pair GEMM: the MMA warp, the epilogue warps of both halves of both CTAs and the commits
on their way, in every order of steps.  Who waits where is read from the kernel's source.  Barriers have phases of one bit, as on the
device: a wait passes when the current phase's parity is the other one."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2by4-pretrain_b200", "csrc", "spmm_sm100.cu")


def _rules():
    src = re.sub(r"//[^\n]*", "", open(SRC).read())
    kernel = src[src.index("\nspmm_pair_kernel("):src.index("\nspmm_split_kernel(")]
    head = re.search(r"int tl = 0;\s*for \(int tile = pair; tile < n_tiles; tile \+= n_pairs, \+\+tl\) \{(.*?)tc_fence_after", kernel, re.S).group(1)
    commit = re.search(r"tc_commit_pair\(([^;]*tmem_full0[^;]*)\);", kernel).group(1)
    one_half = bool(re.search(r"mbar_init\(tmem_empty0 \+ 8 \* b, EPI == EPI_PLAIN \? 8 : 16\)", kernel))
    skips = re.search(r"if \(EPI == EPI_PLAIN && !last && \(tl & 1\) != half\) continue;.*mbar_wait", head, re.S)
    return {"one_half": one_half, "skips": bool(skips), "own_last": "tmem_last0" in head and "tmem_last0" in commit}


def _explore(tiles, plain, rules):
    """What goes wrong in some order of steps: a set of words, empty where nothing does."""
    one_half, skips, own_last = (plain and rules[r] for r in ("one_half", "skips", "own_last"))
    warps = [(cta, half) for cta in (0, 1) for half in (0, 1)]
    is_last = [t >= tiles - 2 for t in range(tiles)]
    takes = [[t for t in range(tiles) if not (skips and not is_last[t] and t % 2 != half)] for _, half in warps]
    reads = [[not (one_half and not is_last[t] and t % 2 != half) for t in range(tiles)] for _, half in warps]
    signals = [[reads[w][t] and not (one_half and is_last[t]) for t in range(tiles)] for w in range(4)]
    need = 2 if one_half else 4

    def barrier(t):     # and the parity that the epilogue waits for
        return (2 + t % 2, 0) if own_last and is_last[t] else (t % 2, t // 2 % 2)

    start = (0, (), (0,) * 8, (0, 0), (0,) * 4, (False,) * 4)      # tiles issued, commits under way, phases done of 4 barriers x 2 CTAs, arrivals, places, reading
    seen, todo, wrong = {start}, [start], set()
    while todo:
        issued, flying, full, arrived, place, reading = todo.pop()
        after = []
        if issued < tiles and (arrived[issued % 2] // need) % 2 != (issued // 2 % 2) ^ 1:
            at_work = [w for w in range(4) if place[w] < len(takes[w]) and takes[w][place[w]] < issued and takes[w][place[w]] % 2 == issued % 2]
            if any(reads[w][takes[w][place[w]]] for w in at_work):
                wrong.add("an accumulator is written while it is wanted")
            after.append((issued + 1, flying + ((issued, 0), (issued, 1)), full, arrived, place, reading))
        for at, (t, cta) in enumerate(flying):                      # commits arrive in any order
            f = list(full)
            f[barrier(t)[0] + 4 * cta] += 1
            after.append((issued, flying[:at] + flying[at + 1:], tuple(f), arrived, place, reading))
        for w, (cta, _) in enumerate(warps):
            if place[w] == len(takes[w]):
                continue
            t = takes[w][place[w]]
            if not reading[w]:
                bar, parity = barrier(t)
                if full[bar + 4 * cta] % 2 != parity:
                    if t >= issued or (t, cta) in flying:
                        wrong.add("a wait passes before its tile is complete")
                    after.append((issued, flying, full, arrived, place, reading[:w] + (True,) + reading[w + 1:]))
            else:
                a = list(arrived)
                a[t % 2] += signals[w][t]
                after.append((issued, flying, full, tuple(a), place[:w] + (place[w] + 1,) + place[w + 1:], reading[:w] + (False,) + reading[w + 1:]))
        if not after and (issued < tiles or any(place[w] < len(takes[w]) for w in range(4))):
            wrong.add("nobody can go on")
        if wrong:
            return wrong
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return wrong


@pytest.mark.parametrize("tiles", range(1, 9))
@pytest.mark.parametrize("plain", [True, False], ids=["plain", "fused"])
def test_no_order_of_steps_stalls_or_reads_early(tiles, plain):
    rules = _rules()
    assert rules["one_half"]
    assert _explore(tiles, plain, rules) == set()


def test_the_model_finds_what_the_rules_prevent():
    """A warp that waits for tiles it does not take can be lapped by two; one that skips them needs barriers of their own for the last
    two, or it may take the other buffer's phase before for them."""
    assert _explore(5, True, {"one_half": True, "skips": False, "own_last": False}) == {"nobody can go on"}
    assert _explore(4, True, {"one_half": True, "skips": True, "own_last": False}) == {"a wait passes before its tile is complete"}
