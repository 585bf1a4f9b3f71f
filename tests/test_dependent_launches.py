"""Kernels launched while the kernel before them still runs may not read what it
writes through the non-coherent path, so none of these buffers is `const
__restrict__` or read by __ldg in the functions of such a kernel."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vulkanexp_gb300", "csrc")

# functions that run after after_previous(), and the buffers that the kernels
# before them in the same update write
READERS = [
    ("blend_shared.cu", ["over_rays", "blend_probes_shared", "k_blend_fp32_shared"], "rays|W|wsum"),
    ("blend_tc.cu", ["blend_tc_tile", "k_blend_tc"], r"rays|prec|wchunks|rowsum"),
    ("wavefront.cu", ["k_shade_classify", "k_shade_front", "k_shade_front_split", "k_shadow"], "hits|front_count|qcount|rays_out"),
]


def function(text, name):
    """From the definition's name to the brace that closes its body."""
    for m in re.finditer(r"\b%s\(" % name, text):
        depth, i = 0, m.end() - 1
        while True:  # the parameter list
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        if not text[i:].lstrip().startswith("{"):
            continue  # a call
        j = text.index("{", i)
        k, depth = j, 0
        while True:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
            if depth == 0:
                return text[m.start():k]
    raise AssertionError("no definition of %s" % name)


@pytest.mark.parametrize("source,names,buffers", READERS)
def test_running_kernels_results_are_read_coherently(source, names, buffers):
    text = open(os.path.join(CSRC, source)).read()
    for name in names:
        body = function(text, name)
        bad = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(?:%s)\b|__ldg\(\s*&?(?:a\.|hits\.)?(?:%s)\b[^)]*\)" % (buffers, buffers), body)
        assert not bad, "%s in %s: %s" % (name, source, bad)
