"""Rules of the tcgen05 kernels that no run shows while all goes well, checked on their sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "torch_dist_ext_b200" / "csrc"
KERNELS = sorted(p.name for p in CSRC.glob("*.cu"))


def _code(name):
    text = (CSRC / name).read_text()
    return re.sub(r"//[^\n]*|/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m.group()), text, flags=re.S)


def _exits_before_barrier(code):
    """(line of the loop, line of the exit) of every work loop that a thread may leave before the loop's first named barrier."""
    found = []
    for barrier in re.finditer(r"tc::named_barrier_sync\(", code):
        stack = []                                   # (position, text in front) of the blocks that are open here
        start = 0
        for m in re.finditer(r"[{}]|;", code[:barrier.start()]):
            if m.group() == "{":
                stack.append((m.end(), code[start:m.start()]))
            elif m.group() == "}" and stack:
                stack.pop()
            if m.group() != ";" or code[start:m.start()].count("(") == code[start:m.start()].count(")"):
                start = m.end()                      # a `;` inside the parentheses of a `for` ends nothing
        loops = [s for s in stack if re.search(r"\bfor \(", s[1])]
        if not loops:
            continue
        begin = loops[-1][0]
        body = code[begin:barrier.start()]
        if "tc::named_barrier_sync(" in body:
            continue                                 # not the first one
        kinds, start = [], 0
        for m in re.finditer(r"[{}]|;|\bbreak;|\breturn;", body):
            if m.group() == "{":
                kinds.append(bool(re.search(r"\b(for|while) \(", body[start:m.start()])))
            elif m.group() == "}":
                kinds.pop()
            elif m.group().startswith("return") or (m.group() == "break;" and not any(kinds)):
                found.append((code.count("\n", 0, begin) + 1, code.count("\n", 0, begin + m.start()) + 1))
            if m.group() != ";" or body[start:m.start()].count("(") == body[start:m.start()].count(")"):
                start = m.end()
    return found


@pytest.mark.parametrize("name", KERNELS)
def test_no_warp_leaves_before_a_named_barrier(name):
    """Warps that meet at a named barrier inside their work loop all get there, also after a wait that ran out: one that
    leaves for the kernel's closing __syncthreads keeps the others at the named barrier for good. (Where all of them take
    the exit together the verdict comes from named_barrier_or; a warp that is `lost` may attend behind the loop.)"""
    code = _code(name)
    late = re.search(r"if \(lost\) \{(.*?)\n    \}\n", code, flags=re.S)
    if late and "tc::named_barrier_sync(" in late.group(1):      # leaves the loop, and attends behind it
        code = re.sub(r"lost = true;\s*break;", lambda m: re.sub(r"[^\n]", " ", m.group()), code)
    shared = re.sub(r"if \(named_barrier_or\([^{]*\{[^}]*\}", lambda m: re.sub(r"[^\n]", " ", m.group()), code)
    assert _exits_before_barrier(shared) == []


def test_aligned_cluster_barriers_gather_the_warp():
    """barrier.cluster.*.aligned is undefined for a warp whose lanes arrive one by one: a lane that skipped a branch, or left a
    loop early, in front of the barrier. The arrive gathers them, the wait follows it at once."""
    sources = {p: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted(CSRC.glob("**/*.cu*"))}
    raw = [(p.name, s[:m.start()]) for p, s in sources.items() for m in re.finditer(r"barrier\.cluster\.arrive[a-z.]*\.aligned", s)]
    assert raw and all(re.search(r"__syncwarp\(\);\s*asm volatile\(\"$", before) for _, before in raw), [n for n, _ in raw]
    for p, s in sources.items():
        calls = len(re.findall(r"tc::cluster_arrive\(\);", s))
        assert calls == len(re.findall(r"tc::cluster_arrive\(\);\s*tc::cluster_wait\(\);", s)) == len(re.findall(r"tc::cluster_wait\(\);", s)), p.name


@pytest.mark.parametrize("name", KERNELS)
def test_tensor_memory_is_fenced_after_a_wait(name):
    """tcgen05 operations are not ordered by an mbarrier alone: between a wait and the next access to tensor memory (a load, a
    store, an MMA) in the text stands a tcgen05.fence::after_thread_sync."""
    code, waited = _code(name), None
    for m in re.finditer(r"mbar_wait(?:_warp)?\(&?(\w+)|fence_after_thread_sync\(\)|tc::(?:tmem_ld|tmem_st|umma)(?!_commit)\w*\s*[<(]", code):
        if m.group().startswith("mbar_wait"):
            waited = code.count("\n", 0, m.start()) + 1
        elif m.group().startswith("fence"):
            waited = None
        else:
            assert waited is None, f"line {code.count(chr(10), 0, m.start()) + 1}: no fence after the wait of line {waited}"


def test_the_gate_of_a_late_operand_is_ordered_before_its_choice():
    """One lane runs the gate and leaves in shared memory which buffer the operand is in; all lanes read that afterwards. A vote
    alone orders no memory between lanes, __syncwarp does."""
    code = re.sub(r"//[^\n]*", "", (CSRC / "include" / "tdx" / "gemm_core.cuh").read_text())
    between = code[code.index("= gate_y();"):code.index("= pick_y();")]
    assert "__syncwarp();" in between


@pytest.mark.parametrize("name,role,first_wait", [
    ("gemm_scaled.cu", "} else if (warp <= 2 && rank == 0) {", "mbar_wait"),
    ("gemm_tcgen05.cu", "} else if (warp == 1) {", ".template issue<"),
])
def test_counted_waits_begin_after_the_previous_kernel(name, role, first_wait):
    """The MMA warps wait for operands with a limit that counts polls. Launched while the previous kernel of the stream still
    runs (a collective that waits seconds for a late peer), they would use the limit up before the operands can come."""
    code = _code(name)
    begin = code.index(role)
    assert "ptx::pdl_wait();" in code[begin:code.index(first_wait, begin)]
