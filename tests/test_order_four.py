"""A start point that leads to a centre of order four, (sqrt(-1), 0): the one
centre whose numerator z = y (1/d - x^2) is 0. The entry points take any point of
the curve as a start."""
import random

import numpy as np
import pytest

from onion_gen_b200 import _native as N
from onion_gen_b200 import filter as F
from onion_gen_b200 import gpu, workloads

P = 2**255 - 19
D = -121665 * pow(121666, -1, P) % P
ORDER = 2**252 + 27742317777372353535851937790883648493
ROOT = pow(2, (P - 1) // 4, P)  # a square root of -1


def add(a, b):
    (x1, y1), (x2, y2) = a, b
    k = D * x1 * x2 * y1 * y2 % P
    return (x1 * y2 + x2 * y1) * pow(1 + k, -1, P) % P, (y1 * y2 + x1 * x2) * pow(1 - k, -1, P) % P


def multiple(oracle, scalar):
    point = oracle.scalar_base_mult((scalar % ORDER).to_bytes(32, "little"))
    x, y, z = (int.from_bytes(point[i:i + 32], "little") for i in (0, 32, 64))
    zi = pow(z, -1, P)
    return x * zi % P, y * zi % P


def start_before(oracle, steps, sign=1):
    """The point from which `steps` additions of 8G lead to (+-sqrt(-1), 0)."""
    x, y = add((sign * ROOT % P, 0), multiple(oracle, -8 * steps))
    return b"".join(v.to_bytes(32, "little") for v in (x, y, 1, x * y % P))


def test_keys_around_it(oracle):
    """y(P +- Q) = +-c s / (q - X), and the oracle's chain passes through it."""
    rng = random.Random(7)
    inv_d = pow(D, -1, P)
    for sign in (1, -1):
        x = sign * ROOT % P
        for m in [1, 2] + [rng.randrange(3, 4000) for _ in range(8)]:
            x2, y2 = multiple(oracle, 8 * m)
            c, q, s = (1 + inv_d) * x % P, pow(D * y2 * y2, -1, P), x2 * pow(1 + x2 * x2, -1, P) % P
            key = c * s * pow(q - x * x, -1, P) % P
            assert key == add((x, 0), (x2, y2))[1] and -key % P == add((x, 0), (-x2 % P, y2))[1]
        keys = oracle.chain_keys_mt(start_before(oracle, 5, sign), 0, 11)
        for i in range(11):
            y = add((x, 0), multiple(oracle, 8 * (i - 5)))[1]
            assert keys[32 * i:32 * i + 32] == y.to_bytes(32, "little")


def survivors(eng):
    offs, keys = eng.advance_raw()
    order = np.argsort(offs)
    return offs[order], keys[order]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["prefix", "wide", "dump", "suffix"])
def test_an_engine_that_meets_it(oracle, device, kind):
    """1152 candidates, the point of order four at each of the first 27: the
    windows are 13 candidates long, so two of them have it for their centre, and
    in the others a neighbour is it."""
    shape = N.EngineConfig(N.SCHEME_PAIRED, 1, 128, 3, 128, 1 if kind == "dump" else 0, 0)
    n = 128 * 3 * 3
    bits = 26 if kind == "wide" else 12
    words = np.random.default_rng(3).integers(0, 2**64, size=2**bits // 64, dtype=np.uint64)
    fs = F.FilterSet.parse_all(["a?", "[b-q]7"] + workloads.suffix_filters(40, 8))
    for steps in range(1, 28):
        start = start_before(oracle, steps, 1 if steps % 2 else -1)
        keys = np.frombuffer(oracle.chain_keys_mt(start, 1, n), dtype=np.uint8).reshape(-1, 32)
        head = keys[:, :4].copy().view(">u4").reshape(-1).astype(np.uint64)
        if kind == "suffix":
            eng = gpu.Engine(device, start, filters=fs, config=shape)
            w, b = fs.index_words()
            slot = head >> np.uint64(32 - b)
            hit = w[slot >> np.uint64(6)] >> (slot & np.uint64(63)) & np.uint64(1)
            w, b = fs.suffix_index_words()
            slot = (keys[:, 24:].copy().view(">u8").reshape(-1).astype(np.uint64) >> np.uint64(1)) & np.uint64(2**b - 1)
            hit |= w[slot >> np.uint64(6)] >> (slot & np.uint64(63)) & np.uint64(1)
        elif kind == "dump":
            eng, hit = gpu.Engine(device, start, config=shape), np.ones(n)
        else:
            eng = gpu.Engine(device, start, bitmap=words, bitmap_bits=bits, config=shape)
            slot = head >> np.uint64(32 - bits)
            hit = words[slot >> np.uint64(6)] >> (slot & np.uint64(63)) & np.uint64(1)
        want = np.nonzero(hit)[0]
        offs, found = survivors(eng)
        eng.close()
        assert len(want) > 20, kind
        assert np.array_equal(offs, 8 * (1 + want.astype(np.uint64))), steps
        assert np.array_equal(found, keys[want]), steps


@pytest.mark.gpu
@pytest.mark.parametrize("dump", [False, True])
def test_a_search_without_allocation_that_meets_it(oracle, device, dump):
    import torch

    lanes, half, rounds, bits = 128, 1, 3, 12
    slots = 2 * half + 1
    n = lanes * slots * rounds
    words = np.random.default_rng(3).integers(0, 2**64, size=2**bits // 64, dtype=np.uint64)
    bitmap = torch.from_numpy(words.view(np.int64)).cuda()
    hits, count = (torch.zeros(k, dtype=torch.int32, device="cuda") for k in (n * 12, 1))
    for steps in range(1, 28):
        start = start_before(oracle, steps)
        keys = np.frombuffer(oracle.chain_keys_mt(start, 1, n), dtype=np.uint8).reshape(-1, 32)
        slot = keys[:, :4].copy().view(">u4").reshape(-1).astype(np.uint64) >> np.uint64(32 - bits)
        hit = np.ones(n) if dump else words[slot >> np.uint64(6)] >> (slot & np.uint64(63)) & np.uint64(1)
        want = np.nonzero(hit)[0]
        err = N.errbuf()
        N.check(N.lib.og_search_noalloc(device.ordinal, start, lanes, half, rounds, None if dump else bitmap.data_ptr(),
                                        bits, hits.data_ptr(), n, count.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream, err, 512), err)
        recs = hits[: int(count.item()) * 12].cpu().numpy().reshape(-1, 12)
        lane, step = recs[:, 0].astype(np.int64), recs[:, 1].astype(np.int64)
        at = (step // slots * lanes + lane) * slots + step % slots
        order = np.argsort(at)
        assert np.array_equal(at[order], want), steps
        assert np.array_equal(np.ascontiguousarray(recs[order, 4:]).view(np.uint8), keys[want]), steps
