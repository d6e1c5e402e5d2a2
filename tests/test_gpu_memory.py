"""Device memory that small searches hold, and that a search in little memory
finds what it does in plenty (-m gpu)."""
import numpy as np
import pytest
import torch

from onion_gen_b200 import _native as N
from onion_gen_b200 import batch as B
from onion_gen_b200 import filter as F
from onion_gen_b200 import gpu, key, workloads

pytestmark = pytest.mark.gpu
MIB = 2**20


def held(make):
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    it = make()
    return it, (before - torch.cuda.mem_get_info()[0]) / MIB


def hits_of(batch, searches):
    for i in range(searches):
        batch.admit(i, workloads.seed(60 + i), ["q7", "ab%s" % "cdef"[i % 4]], 5)
    while batch.running():
        batch.step()
    return [[(h.offset, h.packed) for h in batch.results(i)] for i in range(searches)]


@pytest.mark.parametrize("half,slots,rounds,most", [(5, 256, 1, 300), (5, 256, 40, 330), (64, 8192, 1, 500),
                                                    (64, 0, 1, 1400)])
def test_a_batch_holds_what_its_pool_needs(device, half, slots, rounds, most):
    """Scratch for windows that spread a step over the device, not for the
    longest there are (1.9 GB). The survivors' buffers are 200 MB of this."""
    b, mib = held(lambda: B.Batch(device, half=half, slots=slots, rounds=rounds))
    got = hits_of(b, 3)
    b.close()
    assert mib < most
    other = B.Batch(device, half=256, slots=128 * 300)
    assert hits_of(other, 3) == got
    other.close()


def test_an_engine_stores_two_values_a_group(device):
    """3.9e8 candidates, windows of 430 groups: 64 bytes a group and thread,
    2.1 GB, where room for every key in full is 3.1."""
    words, bits = F.FilterSet.parse_all(["abcdef"]).index_words()
    shape = N.EngineConfig(N.SCHEME_PAIRED, 2048, 94720, 1, 128, 0, 0)
    eng, mib = held(lambda: gpu.Engine(device, key.start_point(workloads.seed(1)), bitmap=words, bitmap_bits=bits,
                                       config=shape))
    eng.close()
    assert mib < 2300


@pytest.mark.parametrize("scheme,half,lanes,rounds,bits,most", [
    (N.SCHEME_PAIRED, 16, 94720, 40, 0, 320), (N.SCHEME_PAIRED, 5, 1024, 2000, 0, 200),
    (N.SCHEME_CHAIN, 4, 94720, 100, 0, 200), (N.SCHEME_PAIRED, 16, 94720, 10, 25, 320)])
def test_an_engine_in_little_memory(device, scheme, half, lanes, rounds, bits, most):
    """With 6 GB free, an engine of a short half holds about what that half's
    own windows take, though its advance is long, and two advances bring what
    they do when memory is plenty."""
    words, bits = F.FilterSet.parse_all(["ab", "q7x"], bits=bits).index_words()
    start, shape = key.start_point(workloads.seed(31)), N.EngineConfig(scheme, half, lanes, rounds, 128, 0, 0)

    def run():
        eng, mib = held(lambda: gpu.Engine(device, start, bitmap=words, bitmap_bits=bits, config=shape))
        out = []
        for _ in range(2):
            offs, keys = eng.advance_raw()
            order = np.argsort(offs)
            out += [offs[order], keys[order]]
        room = eng.room()
        eng.close()
        return out, mib - 2 * 48 * room / MIB

    want, _ = run()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - 6 * 2**30, dtype=torch.uint8, device="cuda")
    try:
        got, mib = run()
    finally:
        del filler
        torch.cuda.empty_cache()
    assert mib < most
    assert all(np.array_equal(a, b) for a, b in zip(got, want)) and len(want[0]) > 100
