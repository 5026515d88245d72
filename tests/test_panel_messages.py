"""The panel leaf's message barriers: which phase is waited for, armed and sent to,
also after a wait has expired, run on the host against a model of an mbarrier."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "rochpl_b200", "csrc")

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("msgs") / "panel_messages")
    subprocess.check_call(["g++", "-std=c++20", "-O1", "-pthread", "-I", CSRC, "-o", exe,
                           os.path.join(HERE, "panel_messages.cpp")])
    return lambda *a: subprocess.run([exe, *map(str, a)], timeout=120).returncode


@pytest.mark.parametrize("ctas,columns", [(1, 70), (2, 33), (4, 200), (16, 96)])
def test_every_column_arrives(model, ctas, columns):
    assert model(ctas, columns, -1, 1) == 0


@pytest.mark.parametrize("lost", [0, 1, 5, 31, 64])
def test_lost_message_leaves_the_barriers_defined(model, lost):
    """A wait that expires is noticed, no phase is armed twice, and no byte count grows
    past its limit in a panel of 1024 columns."""
    assert model(4, 1024, lost, 1) == 0


def test_model_objects_to_arming_regardless(model):
    assert model(4, 1024, 5, 0) == 1
