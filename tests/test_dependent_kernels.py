"""Kernels that are launched beside the one which writes their input (programmatic dependent launch) read activations by plain
loads: the read-only path is for memory that nothing writes while a kernel runs, and an access through a __restrict__ parameter
may be moved across the wait.  Read off the sources: every kernel with a wait, and every function such a kernel may call."""
import glob
import os
import re

import pytest

from tests.conftest import ROOT

KERNELS = sorted(glob.glob(os.path.join(ROOT, "ai-ml-emulation-layer-for-vulkan_b200", "csrc", "kernels", "*.cu*")))
WAIT = re.compile(r"dependencySync\(\)|griddepcontrol\.wait")
# what __ldg may read: RESCALE parameters, tables, border classes, corrections of window convolutions (constant weights) and weight
# tables, all of them constants of the graph or made from such
CONSTANT = re.compile(r"(\w+\.)*(mult|shift|rowClass|colClass|gatherTable|recipTable|residualTable|table)\b|\(?(mult|shift|table|lut|rows|"
                      r"columns|channel)\b|static_cast<const int8_t \*>\(e\.table\)")


def functions(path):
    """(head, body) of every function at the start of a line."""
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for match in re.finditer(r"^(?:template <[^\n]*>\n)?((?:__global__|__device__)[^;{]*?\))\s*\{\n(.*?)^\}", text, re.S | re.M):
        yield match.group(1), match.group(2)


def read_only_arguments(body):
    for match in re.finditer(r"__ldg\(", body):
        depth, at = 1, match.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(body[at], 0)
            at += 1
        yield body[match.end():at - 1]


@pytest.mark.parametrize("path", KERNELS, ids=os.path.basename)
def test_no_read_only_access_to_activations(path):
    waiting = 0
    for head, body in functions(path):
        name = re.findall(r"(\w+)\(", head)[-1]
        if head.startswith("__global__"):
            if not WAIT.search(body):
                continue
            waiting += 1
            assert "__restrict__" not in head, name
        for argument in read_only_arguments(body):
            window = os.path.basename(path) == "gemm_i8_window.cu" and (argument.startswith("p.corr + ") or argument.startswith("own + "))
            assert window or CONSTANT.match(argument), f"{name}: __ldg({argument})"
    text = open(path).read()
    if "launchOverlapped(" in text.replace("inline cudaError_t launchOverlapped(", ""):
        assert waiting > 0, "no kernel with a wait was recognised in a file that launches some"


def test_issuing_warp_of_the_peak_loop_waits_as_a_whole():
    """Its lanes go on to elect.sync together or leave together: no wait decides by the lane."""
    text = open(next(p for p in KERNELS if p.endswith("int8_mma_peak.cu"))).read()
    assert len(re.findall(r"\bmbarWaitWarp\(", text)) == 2 and not re.search(r"\bmbarWait\(", text)


@pytest.mark.gpu
@pytest.mark.parametrize("batches", [1, 2, 3, 4, 65])
def test_peak_loop_of_few_batches(mlel, batches):
    """Batches that need no wait before the drain, one, and several; no wait runs out (checked behind every test)."""
    assert mlel.measure_int8_mma_peak(batches) > 0
