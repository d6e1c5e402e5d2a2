"""The work a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values. ``prepare(case, seed)`` makes what a
program holds before the call (engine, batch, server, device buffers, filter
set), ``run(state)`` is one pass through the public entry points, and
``work(case)`` is what that pass cannot do without. Survivors and matches
come back from the device in no fixed order, so each pass puts them in offset
order, as the run driver does before it takes the first hits, into arrays of
the program's own that hold as many as may come.
"""
from __future__ import annotations

import hashlib
import math
import random
import time

import numpy as np
import torch

from onion_gen_b200 import _native as N
from onion_gen_b200 import batch as B
from onion_gen_b200 import filter as F
from onion_gen_b200 import gpu, key, run as R, serve as S
from onion_gen_b200.workloads import ALPHABET

# lanes of one wave of resident 128-thread blocks (five an SM, 148 SMs)
WAVE = 94720
# unlimited quota of a leased block (run.UNLIMITED)
UNLIMITED = R.UNLIMITED


def listed():
    return [
        # one advance of a small explicit shape, the size of the engine tests:
        # a caller that wants a short answer time, bound by latency
        dict(name="advance_small", kind="advance", half=64, lanes=1024, rounds=4, prefixes=1, lo=3, hi=3, match=False),
        # an odd inversion batch, a lane count that fills no whole wave, several rounds
        dict(name="advance_ragged", kind="advance", half=333, lanes=38272, rounds=3, prefixes=7, lo=4, hi=6,
             match=False),
        # the plain search at the engine's default shape: one 6-symbol prefix,
        # survivors to the host (3.1e9 candidates an advance)
        dict(name="advance_default", kind="advance", half=0, lanes=0, rounds=0, prefixes=1, lo=6, hi=6, match=False),
        # many prefixes, matched on the device (a dense index; half as the
        # default shape picks it for such an index)
        dict(name="match_many", kind="advance", half=512, lanes=2 * WAVE, rounds=1, prefixes=10000, lo=5, hi=8,
             match=True),
        # suffix filters: full keys, sign bit and checksum recomputed on the device
        dict(name="suffix", kind="suffix", half=256, lanes=2 * WAVE, rounds=1, suffixes=16, length=9),
        # the chain scheme at the size of the bit-exact contract: 4096 lanes x 256 steps, one 4-symbol prefix
        dict(name="chain_small", kind="chain", n=256, lanes=4096, rounds=1, prefixes=1, lo=4, hi=4),
        # the chain scheme at four waves of lanes and its default n
        dict(name="chain_large", kind="chain", n=1024, lanes=4 * WAVE, rounds=1, prefixes=1, lo=6, hi=6),
        # a search in buffers of the caller's, nothing allocated
        dict(name="noalloc", kind="noalloc", half=56, lanes=8960, rounds=40, prefixes=1, lo=4, hi=4),
        # a worker's leased range: every block one unlimited search, one step of the batch
        dict(name="lease_step", kind="lease", searches=32, slots=2 * WAVE, half=256, prefixes=100, lo=6, hi=6),
        # a mixed batch of searches from admission to the last quota
        dict(name="batch_quota", kind="quota", searches=24, slots=2 * WAVE, half=256, max_half=2048, most=5000, lo=4,
             hi=5),
        # a burst of requests to the serving loop, until all are answered
        dict(name="serve_burst", kind="serve", searches=48, slots=2 * WAVE, half=256, most=200, lo=4, hi=5),
        # one whole call of the run driver: engine made, quota found, engine closed
        dict(name="search_call", kind="search", half=256, lanes=WAVE, quota=4, prefixes=3, lo=4, hi=5, match=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lanes(rng, lo, hi):
    return max(1, _log(rng, lo, hi) // 128) * 128


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["advance", "advance", "advance", "advance", "suffix", "chain", "chain", "noalloc", "lease",
                       "quota", "serve", "search"])
    if kind in ("advance", "suffix", "search"):
        half = _log(rng, 32, 2048)
        lanes = _lanes(rng, 1024, 8 * WAVE)
        rounds = rng.randint(1, 4)
        while lanes * (2 * half + 1) * rounds > 1.5e9:
            if rounds > 1:
                rounds -= 1
            else:
                lanes = max(1024, lanes // 256 * 128)
        if kind == "suffix":
            return dict(kind=kind, half=half, lanes=lanes, rounds=rounds, suffixes=_log(rng, 1, 40),
                        length=rng.randint(8, 11))
        if kind == "search":
            lanes = min(lanes, 2 * WAVE)
            return dict(kind=kind, half=half, lanes=lanes, quota=rng.randint(1, 16), prefixes=_log(rng, 1, 200),
                        lo=4, hi=rng.randint(4, 5), match=rng.random() < 0.5)
        prefixes = _log(rng, 1, 10000)
        # many prefixes are long ones, matched on the device: what comes back stays what a user can read
        lo = 3 if prefixes < 4 and lanes < 40000 else 4 if prefixes < 50 else 5
        return dict(kind=kind, half=half, lanes=lanes, rounds=rounds, prefixes=prefixes, lo=lo,
                    hi=lo + rng.randint(0, 3), match=prefixes > 100 or rng.random() < 0.3)
    if kind == "chain":
        n = _log(rng, 64, 1500)
        lanes = _lanes(rng, 2048, 4 * WAVE)
        lo = rng.randint(4, 6)
        return dict(kind=kind, n=n, lanes=lanes, rounds=rng.randint(1, 2) if n * lanes < 1e8 else 1,
                    prefixes=_log(rng, 1, 100), lo=lo, hi=lo + rng.randint(0, 1))
    if kind == "noalloc":
        half = _log(rng, 20, 500)
        lanes = _lanes(rng, 256, 16000)
        while lanes * (2 * half + 3) * 64 + half * 96 > 60e6:
            lanes = max(1, lanes // 256) * 128
        return dict(kind=kind, half=half, lanes=lanes, rounds=rng.randint(1, 40), prefixes=_log(rng, 1, 50), lo=4,
                    hi=rng.randint(4, 6))
    slots = rng.choice([1, 2, 3]) * WAVE - 128 * rng.randint(0, 100)
    half = rng.choice([64, 128, 200, 256, 300, 512])
    searches = _log(rng, 4, 64)
    if kind == "lease":
        return dict(kind=kind, searches=searches, slots=slots, half=half, prefixes=_log(rng, 50, 200), lo=6,
                    hi=rng.randint(6, 7))
    if kind == "quota":
        return dict(kind=kind, searches=searches, slots=slots, half=half, max_half=half * rng.choice([1, 2, 4]),
                    most=_log(rng, 2, 5000), lo=4, hi=rng.randint(4, 5))
    return dict(kind=kind, searches=searches, slots=slots, half=half, most=_log(rng, 2, 200), lo=4,
                hi=rng.randint(4, 5))


def _rng(case, seed):
    return random.Random("%d %s" % (seed, case["kind"]))


def _seed32(rng):
    return hashlib.sha256(b"%d" % rng.getrandbits(64)).digest()


def _prefixes(rng, n, lo, hi):
    return ["".join(rng.choice(ALPHABET) for _ in range(rng.randint(lo, hi))) for _ in range(n)]


def _suffixes(rng, n, length):
    """Suffixes whose tail a v3 address can have (a symbol of "aiqy", then "d")."""
    return ["suffix:" + "".join(rng.choice(ALPHABET) for _ in range(length - 2)) + rng.choice("aiqy") + "d"
            for _ in range(n)]


def _searches(rng, n, most, lo, hi):
    """Searches as a batch gets them: (seed, prefixes, quota), counts log-uniform, quotas 1..16."""
    out = []
    for _ in range(n):
        count = max(1, int(math.exp(rng.random() * math.log(most))))
        out.append((_seed32(rng), _prefixes(rng, count, lo, hi), rng.randint(1, 16)))
    return out


def _room(case):
    """Records that the program's arrays hold: the most a pass is expected to bring, and a margin."""
    kind, n = case["kind"], _candidates(case)
    if kind in ("quota", "serve"):
        return 16 * case["searches"]  # the quotas
    if kind == "search":
        return case["quota"]
    if kind == "suffix":
        share = case["suffixes"] * 2.0 ** -16
    elif case.get("match") or kind == "lease":
        share = case["prefixes"] * 32.0 ** -case["lo"]
    else:  # an index is at least 16 bits wide and passes a hundredth at most
        share = min(0.011, case["prefixes"] * max(2.0 ** -16, 32.0 ** -case["lo"]))
    return int(1.25 * n * share) + 2048


def _arrays(case):
    rows = _room(case)
    out = dict(count=np.zeros(1, np.int64), offset=np.zeros(rows, np.int64), key=np.zeros((rows, 32), np.uint8))
    if case["kind"] in ("lease", "quota", "serve"):
        out["search"] = np.zeros(rows, np.int64)
    if case["kind"] in ("lease", "quota", "serve", "search") or case.get("match"):
        out["filter"] = np.zeros(rows, np.int64)
    return out


def prepare(case, seed):
    rng = _rng(case, seed)
    kind = case["kind"]
    device = gpu.look()[0]
    st = dict(case=case, device=device, out=_arrays(case))
    if kind in ("advance", "chain", "noalloc"):
        fs = F.FilterSet.parse_all(_prefixes(rng, case["prefixes"], case["lo"], case["hi"]))
        words, bits = fs.index_words()
        st.update(filters=fs, bits=bits, start=key.start_point(_seed32(rng)))
        if kind == "noalloc":
            cap = _room(case)
            st.update(cap=cap, bitmap=torch.from_numpy(words.view(np.int64)).cuda(),
                      hits=torch.zeros(cap, 12, dtype=torch.int32, device="cuda"),
                      count=torch.zeros(1, dtype=torch.int32, device="cuda"))
            return st
        scheme = N.SCHEME_CHAIN if kind == "chain" else N.SCHEME_PAIRED
        shape = N.EngineConfig(scheme, case["n"] if kind == "chain" else case["half"], case["lanes"], case["rounds"],
                               128, 0, 0)
        st["engine"] = gpu.Engine(device, st["start"], bitmap=words, bitmap_bits=bits, config=shape)
        if case.get("match"):
            st["engine"].match_on_device(fs)
        return st
    if kind == "suffix":
        fs = F.FilterSet.parse_all(_suffixes(rng, case["suffixes"], case["length"]))
        shape = N.EngineConfig(N.SCHEME_PAIRED, case["half"], case["lanes"], case["rounds"], 128, 0, 0)
        st.update(filters=fs, engine=gpu.Engine(device, key.start_point(_seed32(rng)), filters=fs, config=shape))
        return st
    if kind == "search":
        st.update(seed=_seed32(rng), prefixes=_prefixes(rng, case["prefixes"], case["lo"], case["hi"]),
                  shape=N.EngineConfig(N.SCHEME_PAIRED, case["half"], case["lanes"], 1, 128, 0, 0))
        return st
    if kind == "lease":
        batch = B.Batch(device, half=case["half"], slots=case["slots"], rounds=1, max_searches=case["searches"])
        filters = _prefixes(rng, case["prefixes"], case["lo"], case["hi"])
        root = _seed32(rng)
        for block in range(case["searches"]):
            batch.admit(block, key.block_seed(root, block), filters, UNLIMITED)
        st["batch"] = batch
        return st
    st["searches"] = _searches(rng, case["searches"], case["most"], case["lo"], case["hi"])
    if kind == "quota":
        st["batch"] = B.Batch(device, half=case["half"], slots=case["slots"], rounds=1, max_half=case["max_half"])
    else:
        st["server"] = S.Server(device, half=case["half"], slots=case["slots"], rounds=1)
    return st


def _put(out, **arrays):
    """Fills the program's arrays: the records, and nothing behind them."""
    n, before = len(arrays["offset"]), int(out["count"][0])
    for name, values in arrays.items():
        out[name][:n] = values
        out[name][n:before] = 0
    out["count"][0] = n
    return out


def _in_order(out, offsets, packed, filters=None):
    at = np.argsort(offsets, kind="stable")
    more = {} if filters is None else {"filter": filters[at]}
    return _put(out, offset=offsets[at], key=packed[at], **more)


def _put_hits(out, hits, **more):
    return _put(out, offset=np.array([h.offset for h in hits], dtype=np.int64),
                key=np.frombuffer(b"".join(h.public_key for h in hits), dtype=np.uint8).reshape(-1, 32),
                filter=np.array([h.filter for h in hits], dtype=np.int64), **more)


def _put_searches(out, hits):
    return _put_hits(out, hits, search=np.array([h.search_id for h in hits], dtype=np.int64))


def run(state):
    case, out = state["case"], state["out"]
    kind = case["kind"]
    if kind in ("advance", "chain", "suffix"):
        eng = state["engine"]
        if case.get("match"):
            return _in_order(out, *eng.advance_matches_raw())
        if kind == "suffix":
            # a match may take many advances; its program confirms those of
            # this one on the device and keeps the survivors of the next
            matches = eng.advance_matches_raw()[0]
            return _in_order(out, *eng.advance_raw()) | {"matches": len(matches)}
        return _in_order(out, *eng.advance_raw())
    if kind == "noalloc":
        err = N.errbuf()
        N.check(N.lib.og_search_noalloc(
            state["device"].ordinal, state["start"], case["lanes"], case["half"], case["rounds"],
            state["bitmap"].data_ptr(), state["bits"], state["hits"].data_ptr(), state["cap"],
            state["count"].data_ptr(), torch.cuda.current_stream().cuda_stream, err, 512), err)
        recs = state["hits"][:int(state["count"].item())].cpu().numpy()
        slots = 2 * case["half"] + 1
        lane, step = recs[:, 0].astype(np.int64), recs[:, 1].astype(np.int64)
        offsets = 8 * ((step // slots * case["lanes"] + lane) * slots + 1 + step % slots)
        return _in_order(out, offsets, np.ascontiguousarray(recs[:, 4:]).view(np.uint8))
    if kind == "search":
        found, examined, advances = R.device_search(state["device"], state["seed"], state["prefixes"], case["quota"],
                                                    config=state["shape"], device_match=case["match"])
        return _put_hits(out, found) | {"examined": examined, "advances": advances}
    if kind == "lease":
        return _put_searches(out, state["batch"].step())
    if kind == "quota":
        batch, got = state["batch"], []
        for i, (seed, prefixes, quota) in enumerate(state["searches"]):
            batch.admit(i, seed, prefixes, quota)
        while batch.running():
            batch.step()
        for i in range(len(state["searches"])):
            got += batch.results(i)
            batch.retire(i)
        return _put_searches(out, got)
    server, waiting, got = state["server"], len(state["searches"]), []
    for i, (seed, prefixes, quota) in enumerate(state["searches"]):
        server.submit(i, seed, prefixes, quota)
    while waiting:
        done = server.poll()
        waiting -= len(done)
        got += [d.request_id for d in done]
        if not done:
            time.sleep(1e-4)
    return _put_searches(out, [h for i in sorted(got) for h in server.results(i)])


def _candidates(case):
    kind = case["kind"]
    if kind in ("advance", "suffix", "noalloc", "chain"):
        half, lanes = case.get("half"), case["lanes"]
        slots = case["n"] if kind == "chain" else 2 * (half or 2048) + 1
        return (lanes or 8 * WAVE) * slots * (case["rounds"] or 1) * (2 if kind == "suffix" else 1)
    if kind == "lease":
        return case["slots"] // 128 * 128 * (2 * case["half"] + 1)
    # quota over the chance of a match, at the mean of the lengths and counts
    length = (case["lo"] + case["hi"]) / 2
    if kind == "search":
        return case["quota"] * 32.0 ** length / case["prefixes"]
    return case["searches"] * 8.5 * 32.0 ** length / math.sqrt(case["most"])


def work(case):
    """Every candidate's key takes at least one multiplication in GF(2^255-19),
    64 partial products of 32 bits, each a multiplication and an addition.
    Bytes: the prefix index read once, a record written for each hit."""
    n = _candidates(case)
    return {"bytes": 8192.0 + 40.0 * n * 2.0 ** -16, "flops": 128.0 * n}


def exact(case, seed):
    """All outputs are whole numbers and bytes: nothing is rounded."""
    return None
