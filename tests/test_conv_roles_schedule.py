"""Host model of the handshake of the persistent tcgen05 convolutions (k_conv3x3_rows and
k_conv3x3_narrow in csrc/sg_conv.cu), no GPU.

Agents, interleaved at random: the loader (weights that stay, behind wfull; then per
chunk c: wait empty[c % S] from the second use of a stage on, issue its boxes), the
MMA warp (per tile j: wait acce[j % 2] from the third tile on; per chunk: wait full,
issue, commit empty, after the last chunk of a tile commit accf[j % 2]), eight epilogue
warps (per tile: wait accf[j % 2], read, arrive on acce[j % 2]), the copy engine (boxes
complete in any order) and the tensor cores (MMAs and commits complete in order).
Before it returns the loader waits for the boxes it issued last and the MMA warp for the
MMAs it issued last and for its commits to accf: a wait may give up, and the others then
give up too.

A parity wait for phase i passes when the barrier's completed phases have the parity of
i + 1, so it must find i or i + 1 of them.  Checked besides: every run ends, a stage's
boxes land before its MMAs are issued and are not overwritten under them, an accumulator
buffer is read before it is written again, and nothing is in flight when the CTA gives
its shared and tensor memory up.
"""
import random

import pytest

WARPS = 8


class Bar:
    def __init__(self, count=1):
        self.count, self.arrived, self.phases = count, 0, 0

    def arrive(self):
        self.arrived += 1
        assert self.arrived <= self.count
        if self.arrived == self.count:
            self.arrived, self.phases = 0, self.phases + 1

    def passes(self, i):
        assert i <= self.phases <= i + 1, "parity wait would alias"
        return self.phases == i + 1


def last_use(c, i, S):
    """Phase of stage i's barrier after c chunks (the kernels' drain)."""
    return (c - 1 - ((c - 1 - i) % S)) // S


def run(tiles, nk, S, resident, seed, mistake=None, give_up=None):
    rng = random.Random(seed)
    full, empty = [Bar() for _ in range(S)], [Bar() for _ in range(S)]
    accf, acce, wfull = [Bar() for _ in range(2)], [Bar(WARPS) for _ in range(2)], Bar()
    boxes, mmas = [], []                    # in flight
    holds, reads = [None] * S, [0] * S      # chunk in a stage, its MMAs in flight
    tile_in, unread = [None, None], [0, 0]  # tile in an accumulator buffer, warps that have not read it
    weights = [not resident]
    failed = [False]                        # a wait has given up (at the MMA warp's chunk `give_up`)

    def loader():
        issued = 0
        if resident:
            boxes.append(("w", 0, 0))
        for c in range(tiles * nk):
            st = c % S
            while c >= S and mistake != "no_empty_wait" and not empty[st].passes(c // S - 1) and not failed[0]:
                yield
            if failed[0]:
                break
            issued = c + 1
            assert reads[st] == 0, "a stage is overwritten under its MMAs"
            holds[st] = None
            boxes.append(("x", st, c))
            yield
        if mistake == "no_full_drain":
            return
        while resident and not wfull.passes(0):
            yield
        for i in range(min(S, issued)):
            while not full[i].passes(last_use(issued, i, S)):
                yield

    def mma():
        issued = 0
        while resident and mistake != "no_wfull_wait" and not wfull.passes(0):
            yield
        for c in range(tiles * nk):
            j, st, b = c // nk, c % S, (c // nk) % 2
            if c % nk == 0:
                while j >= 2 and mistake != "no_acce_wait" and not acce[b].passes((j - 2) // 2):
                    yield
                assert unread[b] == 0, "an accumulator buffer is overwritten before it was read"
                tile_in[b], unread[b] = j, WARPS
            while mistake != "no_full_wait" and not full[st].passes(c // S):
                yield
            if c == give_up:
                failed[0] = True
                break
            issued = c + 1
            assert holds[st] == c and weights[0], "MMAs before their operands"
            reads[st] += 1
            mmas.append(("mma", st))
            mmas.append(("empty", st))
            if c % nk == nk - 1:
                mmas.append(("accf", b))
            yield
        if mistake == "no_empty_drain":
            return
        for i in range(min(S, issued)):
            while not empty[i].passes(last_use(issued, i, S)):
                yield
        whole = issued // nk  # tiles committed
        for j in range(max(0, whole - 2), whole if failed[0] and mistake != "no_accf_drain" else 0):
            while not accf[j % 2].passes(j // 2):
                yield

    def epilogue():
        for j in range(tiles):
            b = j % 2
            while not accf[b].passes(j // 2) and not failed[0]:
                yield
            if failed[0]:
                return
            assert tile_in[b] == j
            unread[b] -= 1
            yield
            acce[b].arrive()

    agents = [loader(), mma()] + [epilogue() for _ in range(WARPS)]
    for _ in range(200000):
        pick = rng.randrange(len(agents) + 2)
        if pick < len(agents):
            try:
                next(agents[pick])
            except StopIteration:
                agents.pop(pick)
                if not agents:
                    break
        elif pick == len(agents) and boxes:
            kind, st, c = boxes.pop(rng.randrange(len(boxes)))
            if kind == "w":
                weights[0] = True
                wfull.arrive()
            else:
                holds[st] = c
                full[st].arrive()
        elif mmas:
            kind, i = mmas.pop(0)
            if kind == "mma":
                reads[i] -= 1
            else:
                (empty if kind == "empty" else accf)[i].arrive()
    assert not agents, "no progress"
    assert not boxes and not mmas, "in flight when the CTA ends"


@pytest.mark.parametrize("resident", [False, True])
@pytest.mark.parametrize("nk,S", [(1, 1), (1, 2), (1, 6), (2, 2), (3, 5), (9, 4), (18, 8)])  # 9 and 18: a box per tap
def test_the_roles_meet(nk, S, resident):
    for tiles in (1, 2, 3, 5, 8):
        for seed in range(12):
            run(tiles, nk, S, resident, seed)
            run(tiles, nk, S, resident, seed, give_up=seed % (tiles * nk))


@pytest.mark.parametrize("mistake", ["no_empty_wait", "no_full_wait", "no_acce_wait", "no_wfull_wait", "no_full_drain",
                                     "no_empty_drain", "no_accf_drain"])
def test_planted_mistakes_are_caught(mistake):
    """Each wait left out fails on some interleaving; the drains matter once a wait has given up."""
    with pytest.raises(AssertionError):
        for seed in range(400):
            run(4, 2, 2, True, seed, mistake, give_up={"no_accf_drain": 4}.get(mistake, 3) if "drain" in mistake else None)
