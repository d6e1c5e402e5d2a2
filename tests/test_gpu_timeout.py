"""What a wait of the search kernel that runs out does to its engine or batch
(-m gpu). The failure is planted on the host: the kernel itself ends as ever."""
import pytest

from onion_gen_b200 import _native as N
from onion_gen_b200 import batch as B
from onion_gen_b200 import filter as F
from onion_gen_b200 import gpu, key, workloads

pytestmark = pytest.mark.gpu


def refused(status, call, *args):
    with pytest.raises(N.OgError) as e:
        call(*args)
    assert e.value.status == status


@pytest.mark.parametrize("match", [False, True])
def test_an_engine_reports_it_and_closes(device, match):
    fs = F.FilterSet.parse_all(["ab"])
    words, bits = fs.index_words()
    eng = gpu.Engine(device, key.start_point(workloads.seed(1)), bitmap=words, bitmap_bits=bits,
                     config=N.EngineConfig(N.SCHEME_PAIRED, 64, 1024, 1, 128, 0, 0))
    if match:
        eng.match_on_device(fs)
    launch, collect = (eng.launch_matches, eng.collect_matches_raw) if match else (eng.launch, eng.collect_raw)
    launch()
    assert len(collect()[0]) > 0
    launch()
    launch()
    assert N.lib.og_engine_plant_timeout(eng._h) == 0
    refused("OG_E_TIMEOUT", collect)
    refused("OG_E_STATE", launch)
    eng.close()


def test_a_batch_reports_it_and_closes(device):
    b = B.Batch(device, half=64, slots=8192)
    b.admit(1, workloads.seed(1), ["abcdefg"], 1)
    b.step()
    assert N.lib.og_batch_plant_timeout(b._h) == 0
    refused("OG_E_TIMEOUT", b.step)
    refused("OG_E_STATE", b.step)
    refused("OG_E_STATE", b.admit, 2, workloads.seed(2), ["ab"], 1)
    assert b.status(1).done == 0
    b.close()


def test_nothing_to_plant_on():
    assert N.STATUS[N.lib.og_engine_plant_timeout(None)] == "OG_E_ARG"
    assert N.STATUS[N.lib.og_batch_plant_timeout(None)] == "OG_E_ARG"
