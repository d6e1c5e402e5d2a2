"""The engine's timed walk over shapes (-m gpu)."""
import pytest

from onion_gen_b200 import filter as F
from onion_gen_b200 import gpu, key, workloads

pytestmark = pytest.mark.gpu


def test_the_walk_records_one_of_its_shapes(device, tmp_path, monkeypatch):
    """Three halves and three numbers of waves, a lane a thread: what an advance
    covers is all that a shape says."""
    monkeypatch.setenv("ONION_GEN_TUNING_FILE", str(tmp_path / "tuning.yaml"))
    words, bits = F.FilterSet.parse_all(["abcdef"]).index_words()
    start = key.start_point(workloads.seed(5))
    eng = gpu.Engine(device, start, threads=0, bitmap=words, bitmap_bits=bits)
    shape = eng.shape()
    wave = gpu.resident_lanes(device)
    assert shape.half in (512, 1024, 2048) and shape.lanes in (2 * wave, 4 * wave, 8 * wave)
    assert shape.lanes_per_thread == 1 and shape.block == 128
    text = (tmp_path / "tuning.yaml").read_text()
    assert f"first: {shape.half}" in text and f"second: {shape.lanes}" in text
    for s in eng.advance()[:20]:
        key.check_hit(workloads.seed(5), s.offset, s.packed)
