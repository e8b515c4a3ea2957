"""A kernel launched with programmatic stream serialisation lives while the kernel before it still writes. What
that kernel writes must then not be read through the read-only path (__ldg, or a const __restrict__ parameter,
which lets the compiler use it): that path is for data nobody writes during the reader's lifetime, and its
loads may be moved above the wait. It is open only where the kernel before starts its dependents after its last
write, which is when it never says launch_dependents. Checked in the source: the kernels and the names their
bodies use."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gps-pbvr-web_b200", "csrc")

# file, kernel, parameters written by the kernel directly before it, other names of theirs in the body
READS = [
    ("kernels.cu", "k_count_scan", ["cdesc"], []),
    ("kernels.cu", "k_particles", ["etot"], []),
    ("kernels.cu", "k_resolve", ["sub"], []),
    ("sorted.cu", "k_onesweep", ["kin", "vin", "gstart"], []),
    ("denoise.cu", "k_relu_bwd_planes", ["g", "y"], []),
    ("denoise.cu", "k_bias_grad", ["dz"], ["plane"]),
    ("denoise.cu", "k_up2", ["src"], []),
    ("denoise.cu", "k_pool2", ["src"], ["s0"]),
    ("denoise.cu", "k_residual", ["base", "r"], []),
    ("denoise.cu", "k_flip", ["w"], []),
    ("denoise.cu", "k_to_bf16", ["src"], []),
    ("conv3x3.cu", "k_conv3_arrange", ["w"], []),
]


def function(text, name):
    """(parameter list, body) of the definition of `name`."""
    m = re.search(r"\b%s\(([^;{]*)\)\s*\{" % name, text)
    depth, at = 1, m.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
    return m.group(1), text[m.end():at]


@pytest.mark.parametrize("path,kernel,params,aliases", READS, ids=[r[1] for r in READS])
def test_no_read_only_path(path, kernel, params, aliases):
    plist, body = function(source(path), kernel)
    assert "grid_dependency_wait()" in body
    for p in params:
        decl = next(d for d in plist.split(",") if re.search(r"\b%s\s*$" % p, d))
        assert "__restrict__" not in decl, decl
    for name in params + aliases:
        assert not re.search(r"__ldg\((reinterpret_cast<[^>]*>\()?&?\(?%s\b" % name, body), (kernel, name)


def source(name):
    return open(os.path.join(CSRC, name)).read()


def test_read_only_lists_of_a_kernel_that_starts_its_dependents_last():
    # k_particles reads the list through the read-only path
    assert "launch_dependents" not in function(source("kernels.cu"), "k_count_scan")[1]
    # a pass of large tiles reads the one before it that way, a pass of small tiles plainly
    body = function(source("sorted.cu"), "k_onesweep")[1]
    assert body.count("launch_dependents()") == 1 and "if (kEarly) launch_dependents();" in body
    assert body.count("__ldg") == 1 and "kEarly ? *p : __ldg(p)" in body
