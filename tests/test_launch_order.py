"""Order of early launches and tensor memory in the kernels' sources.

A kernel that is launched while its predecessor drains may allocate tensor memory before it waits for that predecessor
(gemm_tc_kernel does).  It then holds columns the predecessor could still be asking for, unless the predecessor lets its
dependents go only once every CTA of its own holds its columns: two such kernels on one SM would wait for one another."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sme_gemm_b200", "csrc")


def _kernels():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\([^{;]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield name, m.group(1), text[m.end():i]


def test_dependents_are_let_go_only_with_tensor_memory_held():
    seen = []
    for name, kernel, body in _kernels():
        allocs = [m.start() for m in re.finditer(r"\btmem_alloc2?\(", body)]
        if not allocs:
            continue
        seen.append(kernel)
        for m in re.finditer(r"\bpdl_launch_dependents\(", body):
            between = body[max(allocs):m.start()] if m.start() > max(allocs) else ""
            assert re.search(r"__syncthreads\(\)|cluster_sync_all\(\)", between), f"{name}: {kernel} lets its dependents go before its CTAs hold tensor memory"
    assert {"gemm_tc_kernel", "attn_tc_kernel", "lowbit_tc_kernel", "lowbit_tc_block_kernel"} <= set(seen)


def test_no_lock_of_the_whole_process_is_held_over_a_launch():
    """A launch waits on the host while its stream's queue is full.  What two launches must be kept together by is the lock of the
    workspace they share (one per device and stream); a lock of the process would keep the threads of every other device waiting."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "api.cu")).read())
    everyones = set(re.findall(r"^(?:static\s+)?std::mutex\s+(\w+);", text, re.M))
    assert everyones
    held = 0
    for m in re.finditer(r"std::(?:lock_guard|unique_lock)<std::mutex>\s+(\w+)\b", text):
        depth, i = 1, m.end()                                      # the rest of the block the lock lives in
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        block = text[m.start():i]
        if not re.search(r"\w+_launch\(", block):
            continue
        held += 1
        locked = re.match(r"[^;]*;[^;]*;", block).group(0)          # the declaration and the statement that locks
        assert not everyones & set(re.findall(r"\w+", locked)), f"{locked.strip()!r} is held over a launch"
    assert held >= 3


def test_words_that_launchers_share_are_atomic():
    """A launcher remembers the device it last raised its kernel's shared-memory limit on, and host threads on several devices read
    and write that word: no function-local static that is written after its initialisation is a plain number."""
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cc")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for kind, word in re.findall(r"^[ \t]+static ([\w:<>]+(?: \w+)*?) (\w+)\s*(?:=\s*-?\d+|\{-?\d+\});", text, re.M):
            seen += 1
            assert kind.startswith("std::atomic<"), f"{name}: static {kind} {word}"
    assert seen >= 7
