"""Rules that the kernels' sources keep and that no run can show reliably."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "infurnace_b200", "csrc")


def test_a_relaxed_arrival_at_a_cluster_barrier_waits_for_what_was_read():
    """A CTA's arrival lets its peers leave or overwrite shared memory that it was reading.  A release orders the reads; a
    relaxed arrival is held back only by a predicate made of the values, and only one that compares them with an operand
    (``%1``): a compiler may know the outcome of a comparison with a constant and drop it."""
    arrivals = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path, encoding="utf-8") as f:
            for line in f:
                for m in re.finditer(r"(@p )?barrier\.cluster\.arrive(\S*)", line):
                    arrivals += 1
                    if ".release" not in m.group(2):
                        assert m.group(1) and re.search(r"setp\.\w+\.s32 p, %0, %1;", line), (os.path.basename(path), line)
    assert arrivals


def test_only_constants_are_read_through_the_read_only_path():
    """A kernel may be resident while the one before it still writes, and a load through ``__ldg`` may be moved ahead of the wait
    for that kernel: it is for what no kernel of a step writes (biases, convolution weights)."""
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path, encoding="utf-8") as f:
            for line in f:
                for m in re.finditer(r"__ldg\(([^)]*)", line):
                    if not m.group(0).endswith("(__ldg"):
                        assert re.search(r"bias|conv_w", m.group(1)), (os.path.basename(path), line)


def test_the_number_of_sms_is_asked_of_the_device_in_one_place():
    """A rule that spreads work goes by the SMs of the device it runs on, not by a number written down."""
    for path in glob.glob(os.path.join(CSRC, "*.c*")) + glob.glob(os.path.join(CSRC, "*.h")):
        with open(path, encoding="utf-8") as f:
            text = f.read()
        assert not re.search(r"\w*SMS?\w*\s*=\s*1\d\d\b", text), os.path.basename(path)
        assert ("cudaDevAttrMultiProcessorCount" in text) == (os.path.basename(path) == "common.cuh"), os.path.basename(path)
