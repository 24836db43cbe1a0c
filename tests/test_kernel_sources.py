"""What the sources of the CUDA kernels promise on every path, where a run cannot show it."""

import re

import pytest

from mfq_b200.ops.build import CSRC

LOADS = re.compile(r"\btmem_ld_\w+\(")


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu*") if p.name != "common.cuh" and LOADS.search(p.read_text())))
def test_no_path_leaves_between_a_tensor_memory_load_and_its_wait(name):
    """Until ``tcgen05.wait::ld`` the registers of a load are the load's, whether its values are used or not: a jump out of the
    sequence would hand them to other values while the load may still write them."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for load in LOADS.finditer(text):
        wait = text.find("tmem_wait_ld()", load.end())
        if wait < 0:  # requested one round ahead: the next round of an unrolled loop begins with the wait
            assert "#pragma unroll" in text[: load.start()] and "tmem_wait_ld()" in text[: load.start()]
            continue
        between = text[load.end() : wait]
        assert not re.search(r"\b(break|continue|return|goto)\b", between), f"{name}:{text.count(chr(10), 0, load.start()) + 1}"


@pytest.mark.parametrize("name", ["fp8_grouped.cu", "fp8_gemm_2cta.cu"])
def test_what_the_kernel_before_wrote_is_not_read_as_constant(name):
    """Under a programmatic launch a grid begins before its inputs are written: only weights may be read through ``__ldg``, which
    promises data that stays the same for the life of the kernel."""
    sources = re.findall(r"__ldg\((?:p\.)?(\w+)", (CSRC / name).read_text())
    assert sources and set(sources) <= {"wsc", "w_scale"}


ALLOCATION = re.compile(r"\btmem_alloc(_pair)?\(")


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu*") if p.name not in ("common.cuh", "pair.cuh") and ALLOCATION.search(p.read_text())))
def test_tensor_memory_is_held_before_a_successor_may_start(name):
    """A successor may allocate before it waits.  Resident beside a CTA that has still to allocate, it could take that CTA's columns and wait
    for its grid for ever, so no path to an allocation passes a trigger, and one comes only after the block barrier behind it."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    kernels = [k for k in text.split("__global__")[1:] if ALLOCATION.search(k)]
    assert kernels
    for kernel in kernels:
        at = ALLOCATION.search(kernel).start()
        for trigger in re.finditer(r"\bpdl_trigger\(\)", kernel[:at]):  # a branch that leaves the kernel without allocating
            depth, end = 0, trigger.end()
            while depth >= 0:
                depth += {"{": 1, "}": -1}.get(kernel[end], 0)
                end += 1
            assert end < at and kernel[:end].rstrip("} \n").endswith("return;"), name
        behind = kernel[at:].find("pdl_trigger()")
        assert behind < 0 or "__syncthreads()" in kernel[at : at + behind], name


def test_an_output_place_is_handed_to_tma_behind_a_proxy_fence():
    """Warps write sums and results to an output place by plain accesses and read them back; what TMA then reads or writes there is only ordered
    behind these by a fence of each thread before the arrival that hands the place over."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "fp8_gemm_2cta.cu").read_text())
    handed = [m.start() for m in re.finditer(r"mbar_arrive\(&turn_done\[", text)]
    assert len(handed) == 2
    for at in handed:  # nothing touches the place between the fence and the arrival
        fence = text.rfind("fence_proxy_async_smem()", 0, at)
        assert fence >= 0 and not re.search(r"\btotal\(|\bturn_in\(|\.shared\.", text[fence:at])


def test_cluster_barriers_ask_nothing_of_the_lanes_of_a_warp():
    """``barrier.cluster.*.aligned`` is undefined for a warp whose lanes come one after the other, and nothing promises that they come together: not
    behind a loop of different lengths, not behind a block barrier or ``__syncwarp()``.  The form without it counts threads."""
    texts = {p.name: p.read_text() for p in CSRC.glob("*.cu*")}
    assert sum("barrier.cluster.wait" in t for t in texts.values()) >= 7
    assert not [n for n, t in texts.items() if re.search(r"barrier\.cluster\.[a-z.]*aligned", t)]


def test_barriers_of_the_grouped_product_have_their_place():
    """What the kernel lays out behind the ring is what the configuration sets aside, for every tile: tiles of 16 tokens have ten stages, and
    their barriers took 264 bytes of 256."""
    text = (CSRC / "fp8_grouped.cu").read_text()
    stages = eval(re.sub(r"BT == (\d+) \? (\d+) :", r"\2 if bt == \1 else", re.search(r"kStages = (BT.*?);", text).group(1)), {"bt": 16})
    acc = int(re.search(r"kAcc = (\d+);", text).group(1))
    fixed = int(re.search(r"turn_free = turn_full \+ (\d+);", text).group(1)) + int(re.search(r"\(turn_free \+ (\d+)\);", text).group(1))
    laid_out = 8 * (2 * stages + 2 * acc + fixed) + 2 * 4
    size = re.search(r"kSmemBytes = kBarsAt \+ (.*?);", text).group(1)
    scope = {"kStages": stages, "kAcc": acc}
    scope["kBarBytes"] = eval(m.group(1), scope) if (m := re.search(r"kBarBytes = (.*?);", text)) else 0
    assert stages == 10 and laid_out <= eval(size, scope) - 1024
