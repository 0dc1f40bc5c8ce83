"""The series that stand for tanh in prompt attention's soft caps (csrc/prefill_attn.cu), as the source states them, against 64 bits."""
import os
import re

import numpy as np
import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmq_b200", "csrc", "prefill_attn.cu")


def series():
    """limit on |z| -> coefficients of z^3, z^5, ... as the kernel rounds them"""
    with open(SOURCE) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    value = {n: np.float32(eval(re.sub(r"(?<=[\d.])f\b", "", e))) for n, e in re.findall(r"\b([tu]\d) = a\.c1 \* (\(?[-+\d. f/e]+\)?)", text)}
    body = text[text.index("auto exponents = "):]
    few, all_ = body.split("} else {")[0], body.split("} else {")[1].split("return")[0]
    limits = re.search(r"z <= ([\d.]+)f\) \? 0 : __all_sync\(0xffffffffu, z <= ([\d.]+)f\) \? 3 : 5", text).groups()

    def order(code):
        return [value[n] for n in sorted(set(re.findall(r"pair_of\(([tu]\d),", code)), key=lambda n: int(n[1:]))]

    return [(float(limits[0]), order(all_)), (float(limits[1]), order(few))]


# where five terms served before, three may not add an error that fp32 would show (2^-24 = 6e-8): a tenth of it.  At the limit of the five
# terms the next one, 1382/155925 z^10, is 5.3e-8.
@pytest.mark.parametrize("which,bound", [(0, 6e-8), (1, 6e-9)])
def test_truncation(which, bound):
    limit, coefficients = series()[which]
    assert len(coefficients) == (4, 2)[which]
    z = np.linspace(limit / 1e5, limit, 100000)
    w, t = z * z, 0.0
    for c in reversed(coefficients):
        t = np.float64(c) + w * t
    # (coefficients rounded to fp32: 2^-25 of the term w / 3 at most)
    assert np.abs((z + z * w * t) / np.tanh(z) - 1).max() < bound + 2.0 ** -25 * limit ** 2 / 3
