"""A batch's items over several rounds and its searches over several steps
(-m gpu): hits from past the first round's candidates and the first step's."""
import pytest

from onion_gen_b200 import _native as N
from onion_gen_b200 import batch as B
from onion_gen_b200 import run, workloads

pytestmark = pytest.mark.gpu

LONG = [["abcde"], ["zzzzz", "qqqqq"]]  # one in 2^25 and one in 2^24
SHORT = [["ab"], ["q7", "zz"], ["cde", "m4"]]


@pytest.mark.parametrize("half,slots,rounds,grid,filters,quotas,item_rounds", [
    # 1.9e9 candidates a step, three rounds an item at 592 CTAs
    (256, 94720, 40, 0, LONG, [45, 90], 3),
    # 3.9e8 a step: two rounds at 148 CTAs
    (256, 94720, 8, 1, LONG, [10, 20], 2),
    # one round an item, many steps
    (5, 256, 3, 0, SHORT, [40, 60, 40], 1),
    (64, 1280, 1, 0, SHORT, [200, 300, 200], 1)])
def test_hits_of_later_rounds_and_steps(device, half, slots, rounds, grid, filters, quotas, item_rounds):
    """The hits of every search are the run driver's, the last of them from
    another round and another step than the first."""
    b = B.Batch(device, half=half, slots=slots, rounds=rounds, grid=grid)
    for i, f in enumerate(filters):
        b.admit(i, workloads.seed(70 + i), f, quotas[i])
    b.step()
    first = [b.status(i).candidates for i in range(len(filters))]  # of the first step
    while b.running():
        b.step()
    big = sum(first) > 1e8
    shape = N.EngineConfig(N.SCHEME_PAIRED, 2048 if big else 256, 94720 if big else 8192, 1, 128, 0, 0)
    for i, f in enumerate(filters):
        want, _, _ = run.device_search(device, workloads.seed(70 + i), f, quotas[i], config=shape)
        got = b.results(i)
        assert [(h.offset, h.public_key, h.filter) for h in got] == [(h.offset, h.public_key, h.filter) for h in want]
        if first[i] == 0:
            continue  # two blocks for three searches: it waited
        at = [h.offset / 8 / first[i] for h in got]  # in steps
        assert at[-1] > 1
        for r in range(item_rounds):
            assert any(r <= item_rounds * a < r + 1 for a in at), (i, r)
    b.close()
