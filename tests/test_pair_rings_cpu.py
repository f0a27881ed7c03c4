"""The two rings of the packed-weight GEMM, as a model of its barriers on the CPU: one loader, two converter
sets that take alternate k blocks, MMAs in order, loads that land in any order.  A wait is the hardware's: it
names the parity of a phase, and holds until the barrier is in a phase of the other parity."""
import ctypes
import random

import pytest

from fluidml_b200 import cabi


class Barrier:
    def __init__(self):
        self.phase = 0

    def over(self, parity):
        return self.phase & 1 != parity & 1


def run(blocks, stages_a, stages_b, rng, common=False):
    """True when every set converts its own blocks and nobody is left waiting.  The sets have a part of A's
    ring each, or (`common`) share all of it."""
    def place(i):
        if common:
            return i % stages_a, i // stages_a
        first, n = (0, (stages_a + 1) // 2) if i % 2 == 0 else ((stages_a + 1) // 2, stages_a // 2)
        return first + (i // 2) % n, (i // 2) // n

    full, empty = [Barrier() for _ in range(stages_a)], [Barrier() for _ in range(stages_a)]
    conv, free = [Barrier() for _ in range(stages_b)], [Barrier() for _ in range(stages_b)]
    holds, flight, wrong = [None] * stages_a, [], []

    def loader():
        for i in range(blocks):
            s, ph = place(i)
            while not empty[s].over(ph ^ 1):
                yield
            flight.append(i)
            yield

    def converter(first):
        for i in range(first, blocks, 2):
            (s, ph), t, pt = place(i), i % stages_b, i // stages_b
            while not full[s].over(ph):
                yield
            if holds[s] != i:
                wrong.append(i)
            empty[s].phase += 1
            while not free[t].over(pt ^ 1):
                yield
            conv[t].phase += 1
            yield

    def mma():
        for i in range(blocks):
            while not conv[i % stages_b].over(i // stages_b):
                yield
            yield
            free[i % stages_b].phase += 1

    def memory():
        done = 0
        while done < blocks:
            if flight:
                i = flight.pop(rng.randrange(len(flight)))
                holds[place(i)[0]] = i
                full[place(i)[0]].phase += 1
                done += 1
            yield

    agents, idle = [loader(), converter(0), converter(1), mma(), memory()], 0
    while agents and idle < 2000 and not wrong:
        a = rng.choice(agents)
        before = [b.phase for b in full + empty + conv + free] + flight
        try:
            next(a)
        except StopIteration:
            agents.remove(a)
        idle = idle + 1 if before == [b.phase for b in full + empty + conv + free] + flight else 0
    return not wrong and not agents


def plan(k, tile_n, split_k, ctas):
    def tensor(rows, cols):
        t = cabi.Tensor()
        t.data, t.rank, t.dtype = 1 << 20, 2, cabi.F32
        t.shape[0], t.shape[1], t.stride[0], t.stride[1] = rows, cols, cols, 1
        return t

    p = cabi.gemm_params(tile_n=tile_n, split_k=split_k)
    p.b_constant, p.b_packed, p.ctas_per_sm = 1, 1 << 21, ctas
    info = cabi.GemmPlanInfo()
    a, b, c = tensor(512, k), tensor(k, 512), tensor(512, 512)
    cabi.check(cabi.lib().fml_gemm_plan(*(ctypes.byref(x) for x in (a, b, c, p, info))))
    return info if info.uses_packed else None


def test_the_model_sees_a_common_ring_of_odd_depth():
    rng = random.Random(1)
    for depth in (3, 5, 7):
        assert not all(run(24, depth, 7, rng, common=True) for _ in range(400))
    assert all(run(24, 4, 7, rng, common=True) for _ in range(400))


@pytest.mark.parametrize("tile_n", [16, 32, 48, 64, 96, 128, 192, 256])
def test_planned_rings(tile_n):
    rng, seen = random.Random(tile_n), set()
    for k in (16, 32, 64, 96, 128, 160, 224, 288, 768, 1024, 4096):
        for split_k in (1, 2, 4, 8):
            for ctas in (1, 2):
                info = plan(k, tile_n, split_k, ctas)
                if info is None:
                    continue
                per = -(-(-(-k // 32)) // split_k)
                assert min(info.stages_a, info.stages) >= 2 or per == 1
                seen.add((min(per, 24), info.stages_a, info.stages))
    assert seen
    for blocks, stages_a, stages_b in seen:
        assert all(run(blocks, stages_a, stages_b, rng) for _ in range(40)), (blocks, stages_a, stages_b)
