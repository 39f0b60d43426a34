"""Orders inside kernels that a run cannot show (a missing wait mostly goes unpunished): read from the sources."""
import re

import pytest

from conftest import ROOT

SOURCES = sorted((ROOT / "pytriton_llama_b200" / "csrc").glob("*.cu*"))


def _kernels(path):
    """(name, body) of every __global__ function of a source, comments left out."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for m in re.finditer(r"__global__", text):
        open_at = text.index("{", m.end())
        depth, at = 1, open_at + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        names = [n for n in re.findall(r"(\w+)\s*\(", text[m.end():open_at]) if n != "__launch_bounds__"]
        yield names[0], text[open_at:at]


KERNELS = [(path.name, name, body) for path in SOURCES for name, body in _kernels(path)]
PEER_ACCESS = re.compile(r"\b(?:st_peer_\w+|ld_peer_\w+|mbar_arrive_cluster|tma_load_2d_pair)\s*\(")


@pytest.mark.parametrize("source,name,body", [k for k in KERNELS if PEER_ACCESS.search(k[2])], ids=lambda v: v if len(v) < 60 else "")
def test_peers_run_before_their_shared_memory_is_touched(source, name, body):
    """The shared memory of another block of a cluster may be used only once that block is known to run: a cluster barrier comes first."""
    waits = [m.start() for m in re.finditer(r"\bcluster_(?:wait|meet)\s*\(", body)]
    assert waits and waits[0] < PEER_ACCESS.search(body).start(), f"{source}: {name}"


@pytest.mark.parametrize("name,inputs", [("token_side_cluster_kernel", ["tokens", "table", "residual"]), ("sample_cluster_kernel", ["logits"]),
                                         ("decode_units_kernel", ["items", "tok_req", "positions"])])
def test_what_a_kernel_of_the_step_may_have_written_is_read_after_the_wait(name, inputs):
    """Reads above the wait on the predecessor are for what no kernel of the step writes; the step's tokens are not (a device kernel
    puts the sampled ones in), nor is what is read by them."""
    body = next(b for _, n, b in KERNELS if n == name)
    for array in inputs:
        read = re.search(rf"\b{array}\s*(?:\[|\+)", body)
        assert read and body.index("pdl_wait()") < read.start(), (name, array)


def test_the_kernels_with_clusters_are_found():
    found = {name for _, name, body in KERNELS if PEER_ACCESS.search(body)}
    assert {"decode_attention_kernel", "gemm_tc_kernel", "sample_cluster_kernel", "token_side_cluster_kernel"} <= found


def _blocks_around(body, at):
    """Where the blocks that hold a place of a kernel's body open, outermost first."""
    opened = []
    for i, c in enumerate(body[:at]):
        if c == "{":
            opened.append(i)
        elif c == "}":
            opened.pop()
    return opened


@pytest.mark.parametrize("source,name,body", [k for k in KERNELS if "pdl_launch_dependents()" in k[2]], ids=lambda v: v if len(v) < 60 else "")
def test_dependents_start_behind_the_wait_on_the_predecessor(source, name, body):
    """A kernel that let its successor start before it has waited itself would have three kernels run side by side, and the successor's
    reads ahead of its wait are right beside its predecessor only: on every path a wait of the same or an enclosing block comes first."""
    for launch in re.finditer(r"pdl_launch_dependents\(\)", body):
        around = _blocks_around(body, launch.start())
        waits = [_blocks_around(body, w.start()) for w in re.finditer(r"(?<=[;{}])\s*pdl_wait\(\);", body[:launch.start()])]
        assert any(w == around[:len(w)] for w in waits), f"{source}: {name}"
