"""Kernels whose launch overlaps the end of the kernel ahead (launch_after in csrc/vrt_device.cuh), by their source:
each begins with its wait, and none reads through the non-coherent path what a kernel ahead of it may still be writing
when its blocks become resident -- that path asks for memory that nothing writes while the kernel runs, and such loads
need not stay below the wait."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "voxelrt_b200" / "csrc"
SOURCES = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*"))}
TEXT = "\n".join(SOURCES.values())
# what no kernel of a frame or of a network call writes: tables uploaded ahead of it, the present table
READ_ONLY = {"lut", "tiles", "firsts"}


def launched():
    names = set(re.findall(r"launch_after\((k_\w+)", TEXT))
    for var, kernel in re.findall(r"auto\* (\w+) = (k_\w+)", TEXT):
        if re.search(r"launch_after\(%s\b" % var, TEXT):
            names.add(kernel)
    return sorted(names)


def definition(name):
    m = re.search(r"__global__[^{;]*?\b%s\(" % name, TEXT)
    assert m, name
    i, depth = m.end(), 1
    while depth:
        depth += {"(": 1, ")": -1}.get(TEXT[i], 0)
        i += 1
    return TEXT[m.end():i - 1], TEXT[TEXT.index("{", i) + 1:]


def test_all_overlapped_kernels_are_found():
    assert {"k_wf_trace", "k_wf_tail", "k_temporal", "k_atrous", "k_b_atrous", "k_present", "k_mlp_grad",
            "k_restir_temporal"} <= set(launched())


@pytest.mark.parametrize("name", launched())
def test_kernel_waits_first_and_reads_coherently(name):
    params, body = definition(name)
    assert body.lstrip().startswith("frame_begin();")
    for p in re.findall(r"const [\w ]+\*\s*__restrict__ (\w+)", params):
        assert p in READ_ONLY, p


@pytest.mark.parametrize("src", ["image_core.cuh", "atrous_tile.cuh", "k_image.cu", "k_atrous.cu", "k_batch.cu", "k_mlp.cu",
                                 "wavefront_core.cuh", "k_restir.cu"])
def test_only_read_only_data_through_the_non_coherent_path(src):
    text = SOURCES[src]
    for arg in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?\s*(\w+(?:\.\w+)*)", text):
        assert arg.split(".")[-1] in READ_ONLY | {"lh", "a"}, arg   # lh: the present table; a: a job table's column
    # pointers that device functions are given on such a kernel's behalf
    for sig in re.findall(r"(?:VRT_DI|__device__ __forceinline__) [\w<>]+ (?:temporal_pixel|atrous_pixel|load_weights|stage_input)"
                          r"\(([^)]*)\)", text):
        assert "__restrict__" not in sig, sig
