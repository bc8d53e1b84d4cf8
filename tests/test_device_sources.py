"""Rules of the device code that a run on a GPU cannot show to be kept, since what breaks them nearly always works: read from the
sources. Needs no GPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "kiln_b200" / "csrc"


def functions(qualifier):
    """(file, name, body) of the functions of that kind."""
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(qualifier + r"\s+(?:[\w:*&<>]+\s+)*(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth, at = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            yield path.name, m.group(1), text[start:at]


KERNELS = {name: (path, body) for path, name, body in functions("__global__")}


def test_the_kernels_are_found():
    assert {"greedy_cluster_kernel", "qlinear_umma_kernel", "attn_kernel", "attn_keys_kernel", "add_rmsnorm_kernel"} <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_peers_have_started_before_their_shared_memory_is_touched(name):
    """CTAs of a cluster may start one after the other: a cluster barrier comes before the first access to another one's memory."""
    body = KERNELS[name][1]
    remote = [m.start() for m in re.finditer(r"shared::cluster|mbar_arrive_cluster\(|cluster_addr\(", body)]
    if remote:
        barrier = [m.start() for m in re.finditer(r"cluster_sync\(\)|cluster_wait\(\)", body)]
        assert barrier and barrier[0] < remote[0]


DEVICE = {}
for _, function, text in functions("__device__ __forceinline__"):
    DEVICE[function] = DEVICE.get(function, "") + text     # overloads together


def test_sums_between_teams_are_stored_as_they_are_polled():
    """What one team leaves in global memory while another one polls it: relaxed stores and loads, never a plain access through the
    pointer."""
    assert "ld.relaxed.gpu" in DEVICE["ql_fix_load"] and "st.relaxed.gpu" in DEVICE["ql_fix_store"]
    for name in ("ql_leave", "ql_go_on"):
        pointers = re.findall(r"uint4\* (\w+) = ql_fix_slot", DEVICE[name])
        assert pointers
        for p in pointers:
            assert not re.search(rf"\b{p}\[|\*{p}\b", DEVICE[name])


@pytest.mark.parametrize("name", ["ql_drain", "ql_drain_wide"])
def test_a_warp_is_whole_before_it_reads_tensor_memory(name):
    """tcgen05.ld is an instruction of the whole warp, and lanes may leave a turn of the loop around it apart."""
    body = DEVICE[name]
    turn = body[body.index("for ("):]
    assert 0 < turn.find("__syncwarp()") < turn.index("tmem_ld")


def test_the_waits_of_the_gemm_are_bounded_by_the_clock():
    """A limit that counts tries is as long as a try happens to be, and one whose start is the kernel's own counts the kernel ahead of
    it, which may itself wait for another GPU: the clock, from that kernel's end."""
    wait = DEVICE["ql_wait"]
    assert 0 < wait.index("griddepcontrol.wait") < wait.index("globaltimer") < wait.index("KC_SPIN_LIMIT_NS")
    assert "KC_SPIN_LIMIT_NS" in DEVICE["mbar_wait"]
    kernel = KERNELS["qlinear_umma_kernel"][1]
    assert not set(re.findall(r"(\w*mbar_\w*wait\w*)\(", kernel)) - {"mbar_test_wait"}
    assert kernel.index("pdl_wait()") < kernel.index("warp_wait(")
