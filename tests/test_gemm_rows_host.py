"""The rule that takes the tiles of csrc/gemm_rows.cu and the launch that it plans for count the same SMs: the device's."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmq_b200", "csrc")


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def test_the_number_of_sms_is_asked_for():
    assert re.findall(r"[^\n]*\b(?:148|74)\b[^\n]*", code("gemm_rows.cu")) == []
    # (what stands for a device that cannot be asked, as on a host without one)
    assert [x.strip() for x in re.findall(r"[^\n]*\b(?:148|74)\b[^\n]*", code("gemm_tcgen05.cu"))] == ["if (n <= 0) n = 148;"]
