"""What no run on one kind of device can show, from the source."""
import re

from conftest import ROOT

ENGINE = (ROOT / "openstc_b200" / "csrc" / "device" / "engine_impl.cuh").read_text()


def test_the_sm_count_is_the_devices_before_anything_is_cut():
    """The launches' cuts follow the SM count, so it is queried first thing in the
    constructor and nowhere replaced by a constant."""
    assert re.findall(r"num_sms_ = (\d+);", ENGINE) == ["0"]
    query = ENGINE.index("cudaDevAttrMultiProcessorCount")
    assert ENGINE.count("cudaDevAttrMultiProcessorCount") == 1
    assert ENGINE.index("explicit EngineT(") < query < ENGINE.index("make_all_tiles();")
