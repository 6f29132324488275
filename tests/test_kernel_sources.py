"""CPU tests of two rules of the kernel sources.  A kernel that is launched while its predecessor still runs
(``griddepcontrol.wait`` inside) must not read what the predecessor writes through loads that the compiler may move
above the wait: parameters that are ``const ... __restrict__``, and the non-coherent ``__ldg`` / ``ld.global.nc``.
Those are for weights.  And a load from TMEM has its wait in the same statement: the registers are not valid before it, and between
two statements the compiler may place anything, a spill of them too."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neurips26-tris-moe_b200", "csrc")
# tables of addresses that the host filled before the first launch
HOST_TABLES = {"peer_recv", "peer_back", "peer_flags"}
PRODUCED = r"row_gather|out_scatter|expert_ids|segment_offsets|num_segments_dev|row_of_flat|selected|perm\b|tok\b|logits|hidden\b|hidden\[|\bx\b|masks|partial"


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(?!__launch_bounds__)(\w+)\s*\(([^{};()]*)\)\s*\{", text, re.S):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield os.path.basename(path), m.group(1), m.group(2), text[m.end():i]


def test_the_sources_are_read():
    names = {name for _, name, _, body in _kernels() if "pdl_wait()" in body}
    assert {"grouped_tiled_kernel", "grouped_decode_kernel", "ep_dispatch_peer_kernel", "combine_routed_kernel"} <= names


@pytest.mark.parametrize("file,name,params,body", [k for k in _kernels() if "pdl_wait()" in k[3]], ids=lambda v: v if isinstance(v, str) and len(v) < 40 else "")
def test_no_movable_load_of_a_predecessors_output(file, name, params, body):
    for p in re.findall(r"const\s+[^,]*?__restrict__\s*(\w+)", params):
        assert p in HOST_TABLES, (file, name, p)
    for load in re.findall(r"(?:__ldg|ldg_stream)\s*\(([^;]*)\)", body):
        assert not re.search(PRODUCED, load), (file, name, load)


def test_a_tmem_load_and_its_wait_are_one_statement():
    loads = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        for asm in re.findall(r"\basm\b[^;]*?\((\s*\"(?:[^\"\\]|\\.)*\".*?)\)\s*;", re.sub(r"//[^\n]*", "", open(path).read()), re.S):
            text = "".join(re.findall(r"\"((?:[^\"\\]|\\.)*)\"", asm))
            if "tcgen05.ld." in text:
                loads += 1
                assert "tcgen05.wait::ld" in text[text.rindex("tcgen05.ld."):], (os.path.basename(path), text[:90])
    assert loads >= 3


def test_the_record_builder_of_a_streamed_layer_waits_for_the_last_use_of_its_place():
    """The layer before may run on another stream, which only the event orders."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "layer.cu")).read())
    body = text[text.index("int tris_moe_layer_forward_paged("):]
    wait = re.search(r"cudaStreamWaitEvent\(s, event\(paged->event_consumed\)", body)
    assert wait and wait.start() < body.index("ahead(0);"), "records are written before their last reader is done"
