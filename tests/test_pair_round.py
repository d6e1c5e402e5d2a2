"""The paired round's arithmetic: one denominator for P + Q and P - Q, and the
low limb of a product without the product.

On the CPU the two identities are checked in Python integers; on a B200
(-m gpu) the survivors of a bitmap that passes half of all slots, which every
candidate's low limb decides, are compared with the oracle's keys."""
import random

import numpy as np
import pytest

from onion_gen_b200 import _native as N
from onion_gen_b200 import filter as F
from onion_gen_b200 import gpu, key, workloads

P = 2**255 - 19
D = -121665 * pow(121666, -1, P) % P
ORDER = 2**252 + 27742317777372353535851937790883648493


def affine(oracle, scalar):
    point = oracle.scalar_base_mult((scalar % ORDER).to_bytes(32, "little"))
    x, y, z = (int.from_bytes(point[i:i + 32], "little") for i in (0, 32, 64))
    zi = pow(z, -1, P)
    return x * zi % P, y * zi % P


def test_both_neighbours_share_a_denominator(oracle):
    rng = random.Random(5)
    for i in range(40):
        s, m = (rng.getrandbits(250), rng.randrange(1, 2049)) if i else (8 * 7, 7)  # the first: P = Q
        x, y = affine(oracle, s)
        x2, y2 = affine(oracle, 8 * m)
        inv_d = pow(D, -1, P)
        z, c = y * (inv_d - x * x) % P, (1 + inv_d) * x % P
        v, q, t = pow(y2, -1, P), pow(D * y2 * y2, -1, P), x2 * pow(1 + x2 * x2, -1, P) % P
        w = pow(q - x * x, -1, P)
        assert (z * v + c * t) * w % P == affine(oracle, s + 8 * m)[1]
        assert (z * v - c * t) * w % P == affine(oracle, s - 8 * m)[1]


def low_product(a, b):
    """The device's low_product: columns 7 and 8, the high halves of column 6
    and of a7 b7, modulo 2^64."""
    x = [(a >> 32 * i) & 0xFFFFFFFF for i in range(8)]
    y = [(b >> 32 * i) & 0xFFFFFFFF for i in range(8)]
    acc = sum(x[i] * y[7 - i] for i in range(8)) + sum(x[i] * y[6 - i] >> 32 for i in range(7))
    acc += (sum(x[i] * y[8 - i] for i in range(1, 8)) << 32) + 38 * (x[7] * y[7] >> 32)
    return acc & (2**64 - 1), x[0] * y[0]


def test_low_product_error_and_low_limb():
    """floor(T / p), from `acc` with at most 128 units of 2^-31 missing, gives
    the low limb of the canonical product, for a sum and a difference too."""
    rng = random.Random(6)
    ends = [0, 1, 2**256 - 1, 2**255, P, 2 * P, 2**256 - 2**224, 2**224 - 1]
    pairs = [(a, b) for a in ends for b in ends] + [(rng.getrandbits(256), rng.getrandbits(256)) for _ in range(3000)]
    sure = 0
    for (a, b), (e, f) in zip(pairs, pairs[1:]):
        (s, lo), (u, mo) = low_product(a, b), low_product(e, f)
        assert ((a * b << 31) // P - s) % 2**64 < 128
        for acc, low, true in ((s + u, lo + mo, a * b + e * f), (s - u - 128, lo - mo, a * b - e * f)):
            if acc % 2**31 < 2**31 - 256:
                sure += 1
                assert (low + 19 * (acc % 2**64 >> 31)) % 2**32 == true % P % 2**32
    assert sure > 5900


@pytest.mark.gpu
@pytest.mark.parametrize("bits,half,lanes,rounds,near", [
    (8, 1, 128, 3, None), (13, 31, 256, 2, None), (16, 127, 384, 2, None), (17, 64, 256, 1, 40), (24, 300, 128, 2, 900),
    (26, 2048, 128, 1, None)])
def test_survivors_of_a_half_set_bitmap(oracle, device, bits, half, lanes, rounds, near):
    """`near`: the start lies so many steps of 8G before the identity, so that
    centres and their neighbours meet it, the table's points and their negatives."""
    start = (oracle.scalar_base_mult(oracle.secret_scalar(workloads.seed(21))) if near is None
             else oracle.scalar_base_mult(((ORDER - 8 * near) % ORDER).to_bytes(32, "little")))
    words = np.random.default_rng(bits).integers(0, 2**64, size=2**bits // 64, dtype=np.uint64)
    eng = gpu.Engine(device, start, bitmap=words, bitmap_bits=bits,
                     config=N.EngineConfig(N.SCHEME_PAIRED, half, lanes, rounds, 128, 0, 0))
    offs, keys = eng.advance_raw()
    n = lanes * rounds * (2 * half + 1)
    all_keys = np.frombuffer(oracle.chain_keys_mt(start, 1, n), dtype=np.uint8).reshape(-1, 32)
    slot = all_keys[:, :4].copy().view(">u4").reshape(-1).astype(np.uint64) >> np.uint64(32 - bits)
    want = np.nonzero((words[slot >> np.uint64(6)] >> (slot & np.uint64(63))) & np.uint64(1))[0]
    order = np.argsort(offs)
    assert np.array_equal(offs[order], 8 * (1 + want.astype(np.uint64)))
    assert np.array_equal(keys[order], all_keys[want])


@pytest.mark.gpu
@pytest.mark.parametrize("scheme,half,lanes,rounds,block", [
    (N.SCHEME_PAIRED, 37, 416, 3, 32), (N.SCHEME_PAIRED, 2048, 128, 1, 128), (N.SCHEME_CHAIN, 1, 128, 1, 128),
    (N.SCHEME_CHAIN, 333, 192, 2, 96), (N.SCHEME_CHAIN, 64, 1024, 1, 128)])
def test_tiled_advances_meet_without_gap(oracle, device, scheme, half, lanes, rounds, block):
    """However an advance is tiled, two in a row bring the same survivors as
    the oracle's keys over both ranges: none past the end of an advance, none
    missing at the seam."""
    start = oracle.scalar_base_mult(oracle.secret_scalar(workloads.seed(22)))
    words = np.random.default_rng(half).integers(0, 2**64, size=2**14 // 64, dtype=np.uint64)
    eng = gpu.Engine(device, start, bitmap=words, bitmap_bits=14,
                     config=N.EngineConfig(scheme, half, lanes, rounds, block, 0, 0))
    slots, first = (2 * half + 1, 1) if scheme == N.SCHEME_PAIRED else (half, 0)
    assert eng.batch() == eng.threads() * rounds * slots
    got = [eng.advance_raw() for _ in range(2)]
    n = 2 * eng.batch()
    all_keys = np.frombuffer(oracle.chain_keys_mt(start, first, n), dtype=np.uint8).reshape(-1, 32)
    slot = all_keys[:, :4].copy().view(">u4").reshape(-1).astype(np.uint64) >> np.uint64(18)
    want = np.nonzero((words[slot >> np.uint64(6)] >> (slot & np.uint64(63))) & np.uint64(1))[0]
    offs, keys = (np.concatenate([g[i] for g in got]) for i in range(2))
    order = np.argsort(offs)
    assert np.array_equal(offs[order], 8 * (first + want.astype(np.uint64)))
    assert np.array_equal(keys[order], all_keys[want])


@pytest.mark.gpu
def test_an_advance_beyond_the_lane_state(device):
    """4.3e10 candidates, more windows than the lane state holds: every lane
    runs two rounds. The survivors are as many as the index lets through, inside
    the range and distinct, and a sample of them re-derives."""
    seed = workloads.seed(23)
    fs = F.FilterSet.parse_all(["qqqq"])
    words, bits = fs.index_words()
    eng = gpu.Engine(device, key.start_point(seed), bitmap=words, bitmap_bits=bits,
                     config=N.EngineConfig(N.SCHEME_PAIRED, 2048, 1 << 20, 10, 128, 0, 0))
    n = eng.batch()
    offs, keys = eng.advance_raw()
    mean = n * fs.occupancy()
    assert abs(len(offs) - mean) < 6 * mean**0.5
    assert offs.min() >= 8 and offs.max() <= 8 * n and len(np.unique(offs)) == len(offs)
    order = np.argsort(offs)
    for i in order[:: len(order) // 100]:
        key.check_hit(seed, int(offs[i]), bytes(keys[i]))
    assert offs[order[0]] < 8 * n * 1e-4 and offs[order[-1]] > 8 * n * 0.9999


@pytest.mark.gpu
@pytest.mark.parametrize("half,lanes,rounds", [(1, 128, 1), (56, 8960, 40), (200, 2432, 31), (2048, 128, 3)])
def test_search_without_allocation_in_several_rounds(device, half, lanes, rounds):
    """The search in the fixed array finds what an engine of the shape does,
    numbered in the caller's lanes and steps, whether its tiling takes one round
    or many."""
    import torch

    start = key.start_point(workloads.seed(24))
    words, bits = F.FilterSet.parse_all(["ab", "q7x", "mm"]).index_words()
    slots = 2 * half + 1
    n = lanes * rounds * slots
    cap = n // 64 + 4096
    bitmap = torch.from_numpy(words.view(np.int64)).cuda()
    hits, count = (torch.zeros(k, dtype=torch.int32, device="cuda") for k in (cap * 12, 1))
    err = N.errbuf()
    N.check(N.lib.og_search_noalloc(device.ordinal, start, lanes, half, rounds, bitmap.data_ptr(), bits, hits.data_ptr(),
                                    cap, count.data_ptr(), torch.cuda.current_stream().cuda_stream, err, 512), err)
    recs = hits[: int(count.item()) * 12].cpu().numpy().reshape(-1, 12)
    lane, step = recs[:, 0].astype(np.int64), recs[:, 1].astype(np.int64)
    assert lane.size == 0 or (lane.max() < lanes and step.max() < rounds * slots)
    got = 8 * ((step // slots * lanes + lane) * slots + 1 + step % slots)
    eng = gpu.Engine(device, start, bitmap=words, bitmap_bits=bits,
                     config=N.EngineConfig(N.SCHEME_PAIRED, half, lanes, rounds, 128, 0, 0))
    want, keys = eng.advance_raw()
    a, b = np.argsort(got), np.argsort(want)
    assert np.array_equal(got[a], want[b].astype(np.int64)) and len(got) > n // 1000
    assert np.array_equal(np.ascontiguousarray(recs[a, 4:]).view(np.uint8), keys[b])


@pytest.mark.gpu
@pytest.mark.parametrize("prefixes,suffixes,length", [([], 40, 8), (["ab", "q7x"], 16, 9), (["m"], 3, 11)])
def test_survivors_of_suffix_and_prefix_bitmaps(oracle, device, prefixes, suffixes, length):
    """The survivors of a filter engine are the candidates whose slot is set in
    either bitmap, over two advances."""
    fs = F.FilterSet.parse_all(prefixes + workloads.suffix_filters(suffixes, length))
    start = oracle.scalar_base_mult(oracle.secret_scalar(workloads.seed(25)))
    eng = gpu.Engine(device, start, filters=fs, config=N.EngineConfig(N.SCHEME_PAIRED, 100, 3712, 2, 128, 0, 0))
    n = 2 * eng.batch()
    keys = np.frombuffer(oracle.chain_keys_mt(start, 1, n), dtype=np.uint8).reshape(-1, 32)
    hit = np.zeros(n, dtype=bool)
    tail = keys[:, 24:].copy().view(">u8").reshape(-1).astype(np.uint64) >> np.uint64(1)
    words, bits = fs.suffix_index_words()
    slot = tail & np.uint64(2**bits - 1)
    hit |= (words[slot >> np.uint64(6)] >> (slot & np.uint64(63)) & np.uint64(1)).astype(bool)
    if prefixes:
        words, bits = fs.index_words()
        slot = keys[:, :4].copy().view(">u4").reshape(-1).astype(np.uint64) >> np.uint64(32 - bits)
        hit |= (words[slot >> np.uint64(6)] >> (slot & np.uint64(63)) & np.uint64(1)).astype(bool)
    want = np.nonzero(hit)[0]
    got = [eng.advance_raw() for _ in range(2)]
    offs, found = (np.concatenate([g[i] for g in got]) for i in range(2))
    order = np.argsort(offs)
    assert len(want) > 200 and np.array_equal(offs[order], 8 * (1 + want.astype(np.uint64)))
    assert np.array_equal(found[order], keys[want])
