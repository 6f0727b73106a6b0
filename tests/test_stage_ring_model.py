"""No bulk copy is in flight when a CTA of the training kernels exits after a
wait of its own ran out: the drain's chunks and parities (stage_ring.hpp, which
the kernels use) on a model of the mbarriers, with the copies landing in every
order."""
import re
import subprocess

from conftest import ROOT

CSRC = ROOT / "openstc_b200" / "csrc"


def test_abandoned_copies_are_waited_for(tmp_path):
    exe = tmp_path / "ring"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), str(ROOT / "tests" / "stage_ring_model.cpp"), "-o",
                    str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr


def test_training_kernels_drain_what_they_started():
    """Each ring is drained by its own slot count and by the chunks it started,
    and the MMAs' last commit does not depend on the waits."""
    text = (CSRC / "device" / "mlp_train.cuh").read_text()
    rings = re.findall(r"using Ring = tc::StageRing<(\w+)>", text)
    assert rings == re.findall(r"drain<(\w+)>\(full, issued\)", text) == ["2", "kDwStages"]
    assert "if (ok) tc::commit" not in text
