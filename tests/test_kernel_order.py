"""Order of instructions in kernels that hold tensor memory or copies in flight, read from their sources: what it guards against
cannot be shown by running it (a grid that waits for another one without a limit, a copy that lands after its block has left)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "runit_mac_b200" / "csrc"


def kernels(path):
    """(name, body) of every __global__ function of a source file, comments removed."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
        at = text.index("{", text.index(")", m.end()))
        depth, i = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        yield m.group(1), text[at:i]


def device_functions(path):
    """(name, body) of every kernel, device function and constructor of a source file or header, comments removed."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for m in re.finditer(r"__(?:global|device)__[^;{}]*?\b(\w+)\s*\([^(){};]*\)\s*(?=\{)", text):
        depth, i = 0, m.end()
        while True:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        yield m.group(1), text[m.end():i]


def test_dependents_are_released_after_tensor_memory_is_held():
    """tcgen05.alloc waits without a limit.  A kernel that allocates may let a dependent grid start only when all of its own blocks
    hold their columns: else a block of the dependent grid, which allocates before it waits for its predecessor, can take the columns
    that the predecessor still waits for."""
    seen = set()
    for path in sorted(CSRC.glob("*.cu*")):
        for name, body in device_functions(path):
            alloc, trigger = re.search(r"\btmem_alloc(_pair)?\(", body), body.find("grid_launch_dependents(")
            if not alloc:
                continue
            seen.add(name)
            if trigger < 0:
                continue
            barrier = re.compile(r"__syncthreads\(\)|cluster_sync\(\)").search(body, alloc.end())
            assert barrier and trigger > barrier.end(), "%s (%s) releases its dependents before its allocation is known to be done" % (name, path.name)
    # Block: the constructor that the kernels over tc_rows.cuh begin with; nothing else of theirs may release dependents
    assert seen == {"attention_tc_kernel", "gemm_tc_kernel", "gemm_pair_kernel", "grouped_gemm_pair_kernel", "Block"}
    for source, users in (("gemv_tc.cu", 1), ("moe_slots.cu", 1)):
        bodies = [body for _, body in kernels(CSRC / source) if "tcr::Block<" in body]
        assert len(bodies) == users and not any("grid_launch_dependents(" in b for b in bodies)


@pytest.mark.parametrize("source", ["attention_tc.cu", "moe_slots.cu", "gemv_tc.cu", "gemm_bf16.cu", "moe_grouped.cu"])
def test_copies_in_flight_are_waited_for(source):
    """A role that gives up a bounded wait must not leave with its bulk copies (or MMAs) in flight: they would arrive in shared (tensor)
    memory that belongs to another block by then."""
    seen = 0
    for name, body in kernels(CSRC / source):
        loads = [m.start() for m in re.finditer(r"\b(tma_load_\dd|bulk_load_1d)\(", body)]
        loads = loads or [m.start() for m in re.finditer(r"\btma_load_2d_pair\(", body)]
        if loads:
            seen += 1
            assert body.find("mbar_drain(", loads[-1]) > 0, "%s leaves copies in flight when it gives up" % name
            # whether anyone has given up is known when all roles have ended, and not when the copying one has
            assert "given_up" not in body, name
    assert seen


@pytest.mark.parametrize("source,count", [("attention_tc.cu", 1), ("tc_rows.cuh", 1), ("gemm_bf16.cu", 2), ("moe_grouped.cu", 1)])
def test_products_in_flight_are_waited_for(source, count):
    """Likewise for MMAs: tensor memory goes back when every one that was issued is over."""
    text = re.sub(r"//[^\n]*", "", (CSRC / source).read_text())
    commits = [m.end() for m in re.finditer(r"umma_commit(_pair)?\((last \? done : o_full|drain \+ 8 \* w|bar_mma)", text)]
    assert len(commits) == count
    for at in commits:
        wait = re.compile(r"mbar_wait(_timed)?\((done|drain \+ 8 \* w|bar_mma), 0").search(text, at)
        assert wait and "umma_commit" not in text[at:wait.start()] and "tmem_dealloc" not in text[at:wait.start()]
        if "drain" in wait.group():
            assert not re.search(r"if \(!ok\) \{[^}]*$", text[:at])


def test_clears_are_ordered_with_the_stream():
    """cudaMemset runs on the legacy stream, for which a context's non-blocking stream does not wait: a launch could find tickets or partial
    sums while they are being cleared."""
    for path in sorted(CSRC.glob("*.cu*")):
        assert not re.search(r"\bcudaMemset\(", re.sub(r"//[^\n]*", "", path.read_text())), path.name


def body_after(text, pattern):
    """The braces that follow the first match of a pattern."""
    m = re.search(pattern, text)
    at = i = text.index("{", m.end())
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[at:i]


@pytest.mark.parametrize("role", ["products", "unpack", "sums"])
def test_bounded_waits_begin_behind_the_dependency_wait(role):
    """A dependent grid may be resident while its predecessors still run, for any time: a role that counts that time towards its limit gives up
    on work that is in order.  (A first piece of Q6_K weights is waited for ahead of it: its copies depend on nothing.)"""
    text = re.sub(r"//[^\n]*", "", (CSRC / "tc_rows.cuh").read_text())
    body = body_after(text, r"__device__ __forceinline__ void %s\(" % role)
    assert 0 <= body.find("grid_dependency_wait()") < body.find("wait(", body.find("grid_dependency_wait()") + 22)
    assert not re.search(r"!wait\(", body[:body.index("grid_dependency_wait()")])
    if role == "unpack":
        loop = body[body.index("for (uint32_t e"):]
        assert re.search(r"C::kQ6 && e >= C::kTeams && e < 2 \* C::kTeams\) grid_dependency_wait\(\)", loop[:loop.index("!wait(")])
