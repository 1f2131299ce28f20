"""Rules on the kernels' sources whose breach shows on a GPU only now and then, or harms more than the process: read, not run."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gpustack_b200" / "csrc"
SOURCES = sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), *CSRC.glob("*.h")])


def _instructions(text):
    """PTX instruction names of a source, string pieces of one statement joined."""
    return re.findall(r"cp\.async\.bulk[\w.:]*", re.sub(r'"\s*\n?\s*"', "", text))


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_bulk_copies_go_to_one_cta(path):
    """The library serves several GPUs, whose buffers may be one another's: no bulk copy spreads over a cluster."""
    assert not [i for i in _instructions(path.read_text()) if "multi" + "cast" in i]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_instructions_of_whole_warps_stay_in_place(path):
    """An instruction that waits for other lanes is volatile: the compiler neither moves it into a branch nor makes two of it."""
    text = path.read_text()
    for m in re.finditer(r"\basm\b(?P<v>\s*volatile\b)?\s*\((?P<code>(?:\s*\"[^\"]*\")+)", text):
        if re.search(r"\.sync\b", m["code"]):
            assert m["v"], m["code"]


def _definitions(text):
    """The source cut at every definition that begins a line."""
    return re.split(r"\n(?=template |__global__|__device__|static |extern )", text)


@pytest.mark.parametrize("path", [p for p in SOURCES if p.suffix == ".cu"], ids=lambda p: p.name)
def test_clusters_meet_before_remote_accesses(path):
    """Another CTA's shared memory may be addressed only once that CTA is known to have started."""
    for body in _definitions(path.read_text()):
        if "mapa_u32(" in body:
            assert "cluster_sync_all()" in body and body.index("cluster_sync_all()") < body.index("mapa_u32("), body[:200]


@pytest.mark.parametrize("name", ["moe.cu", "moe_biased.cu"])
def test_routing_reads_earlier_outputs_past_l1(name):
    """A grid that became resident early has missed the launch-time L1 invalidation: what the kernels before it wrote (all of the
    routing kernels' inputs but the weights) is not read by plain loads."""
    kernels = [d for d in _definitions((CSRC / name).read_text()) if "pdl_wait();" in d]
    assert kernels
    for body in kernels:
        head, code = body.split("pdl_wait();", 1)
        for arg in set(re.findall(r"const (?:\w+)\s*\*\s*(?:__restrict__\s+)?(\w+)", head)) - {"correction", "router"}:
            assert not re.search(r"(?<![\w.])%s\[|[ (!]\*%s\b|(?<!_cg_)(?<!rb_)ld_v4\(%s\b" % (arg, arg, arg), code), (arg, body[:120])


def test_chunk_weights_are_read_before_their_buffer_is_free():
    """The state's converting warps read an item's weights only before they hand its last half over: behind that, the weights of the item
    after next take the buffer's place."""
    kernel = next(d for d in _definitions((CSRC / "chunk_tc.cuh").read_text()) if "ct_state_kernel" in d)
    converting = kernel[kernel.index("if (warp < kCtConvWarps)"):kernel.index("else if (warp < kCtConvWarps + kCtReadWarps)")]
    before, behind = converting.split("ct_stored(&half_full[e]);")
    assert re.search(r"\bsc\.w\[", before) and not re.search(r"\b(sc|scratch)\b", behind)


def test_rows_are_copied_once_every_lane_has_read_the_ones_before():
    """A helper warp's lanes read a block's values in turns of their own number and copy the next rows over them, other lanes' columns
    too: the warp meets in between."""
    kernel = next(d for d in _definitions((CSRC / "gated_scan.cu").read_text()) if "\ngated_scan_kernel(" in d)
    read, copy = kernel.index("put(st - AHEAD);"), kernel.index("stage(st - AHEAD + BUFS);")
    between = kernel[read:copy]
    assert read < copy and "__syncwarp();" in between and between.index("__syncwarp();") < between.index("if (")
