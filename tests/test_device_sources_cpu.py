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


# kernel or what it calls -> what kernels before it wrote, by the names under which it reads it
EARLIER = [("chunk_scan.cuh", "chunk_carry_kernel", ["a.ws"]), ("gated_linear_attn.cu", "gla_scan_kernel", ["x", "z"]),
           ("gated_linear_attn.cu", "gla_step_kernel", ["x", "z"]), ("gated_linear_attn.cu", "struct GatedLinearForm", ["p.z", "row"]),
           ("gated_scan.cu", "struct StateSpaceForm", ["p.gates", "row"]), ("gated_scan.cu", "gated_scan_kernel", ["a.gates", "a.x"]),
           ("gated_scan.cu", "gated_step_kernel", ["a.gates", "a.x"]), ("gated_scan.cu", "gate_norm_kernel", ["y", "proj"]),
           ("gated_scan.cu", "gate_norm_heads_kernel", ["y", "proj"]), ("gated_scan.cu", "gate_norm_parts_kernel", ["y", "proj"]),
           ("gemm_simt.cu", "gemm_simt_kernel", ["X"]), ("latent.cu", "latent_prep_rows_kernel", ["proj", "q"]),
           ("latent_attention_mma.cu", "latent_attn_step_kernel", ["a.qa"]), ("latent_attention_mma.cu", "latent_attn_merge_kernel", ["ws"]),
           ("rot_prep.cu", "rot_prep_vec_kernel", ["a.proj"]), ("rot_prep.cu", "rot_plain_kernel", ["a.proj"]),
           ("conv_rec_prep.cu", "conv_rec_prep_vec_kernel", ["a.proj"]), ("conv_prep.cuh", "conv_before", ["src"]),
           ("conv_prep.cuh", "conv_window", ["src"]), ("conv_prep.cuh", "conv_ring_put", ["src"])]


@pytest.mark.parametrize("file,name,wrote", EARLIER, ids=lambda v: v if isinstance(v, str) else "")
def test_early_kernels_read_earlier_outputs_past_l1(file, name, wrote):
    """The same for the kernels of recurrent and latent layers, through every pointer that is formed from such a buffer."""
    text = (CSRC / file).read_text()
    if name.startswith("struct "):
        body = text[text.index(name + " {"):]
        body = body[:body.index("\n};")]
    else:
        body = next(d for d in _definitions(text) if re.search(r"\b%s\(" % name, d) and "{\n" in d)
        body = body[body.index("{\n"):]
    if name == "rot_prep_vec_kernel":                   # the one left with plain loads: nothing released early, no promise that nobody writes
        assert "pdl_wait_in_place();" in body and "__restrict__" not in text and "__ldg(" not in body
        return
    names = list(wrote)
    for m in re.finditer(r"(?:const )?\b(?:float|bf16|TA|TX|uint4)\s*\*\s*(\w+) = ([^;]*);", body):
        if any(re.search(r"(?<![\w.])%s\b" % re.escape(n), m[2]) for n in names):
            names.append(m[1])
    for n in names:
        n = r"(?<![\w.>])" + re.escape(n)
        assert not re.search(n + r"\[", body) and not re.search(r"= \*" + n + r"\b", body) and not re.search(r"\*\s*reinterpret_cast<const [^>]*>\(" + n + r"\b", body) \
            and not re.search(r"(?<!_cg_)\bld_v4\(" + n + r"\b|__ldg\(" + n + r"\b", body), (n, body[:160])


def test_every_early_kernel_is_under_the_rule():
    """Each kernel of these files that waits for the launch before is listed above."""
    listed = {n for _, n, _ in EARLIER}
    for file in {f for f, _, _ in EARLIER}:
        for d in _definitions((CSRC / file).read_text()):
            m = re.search(r"\b(\w+_kernel)\([^;]*?\{\n(?:.*\n)*?.*\b(?:pdl_wait|pdl_wait_in_place|cs_wait_before)\(\);", d)
            if m and "__global__" in d:
                assert m[1] in listed or m[1] in ("chunk_state_kernel", "chunk_output_kernel"), m[1]      # (rows by cp.async.cg, gates by the forms)


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
