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


def test_the_autotuner_times_the_stages_of_the_step():
    """Laminar air has no source stage and starts dq in the flux kernel: the timed
    pass launches the right-hand side as the step does."""
    body = ENGINE[ENGINE.index("double time_stages(int reps)"):]
    body = body[:body.index("pass();")]
    assert "launch_rhs();" in body and "launch_source();" not in body and "launch_flux(" not in body
    residual = ENGINE[ENGINE.index("void launch_residual() {"):ENGINE.index("void launch_rhs() {")]
    assert "launch_rhs();" in residual
