"""Source check of the kernels launched programmatically (csrc/pdl.cuh): such
a kernel may start before the launch ahead of it has finished, so no load of
what that one wrote may be of a kind that the compiler can move above the
wait. Fields that only set-up writes (flags and what is derived from them) are
complete before a step's first launch and may be read in any way."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "foil_cfd_gb300" / "csrc"
STATIC = {"kind", "ckind", "fkind", "codes", "targets", "w"}   # w: the network's weights of the wall update
# Read through the storage's load, which is volatile unless it says otherwise.
POPULATIONS = {"src", "f", "ff"}


def code(path):
    s = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", s)


def block(s, at):
    depth = 0
    for i in range(at, len(s)):
        depth += {"{": 1, "}": -1}.get(s[i], 0)
        if depth == 0 and s[i] == "}":
            return s[at:i + 1]
    raise AssertionError("unbalanced braces")


def kernels():
    for path in sorted(CSRC.glob("*.cu*")):
        s = code(path)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", s):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(s[i], 0)
                i += 1
            body = block(s, s.index("{", i))
            if "griddepcontrol" in body or "pdl_wait" in body:
                yield f"{path.name}:{m.group(1)}", s[m.end():i - 1], body


KERNELS = list(kernels())


def test_every_kernel_launched_so_is_found():
    launched = set()
    for path in CSRC.glob("*.cu*"):
        launched |= set(re.findall(r"\b(\w+_kernel)\b(?=[<,\s])", " ".join(
            re.findall(r"launch_pdl\(.*?;", code(path), flags=re.S))))
    names = {k.split(":")[1] for k, _, _ in KERNELS}
    assert launched and launched <= names
    assert len(KERNELS) >= 15


@pytest.mark.parametrize("name,params,body", KERNELS, ids=[k for k, _, _ in KERNELS])
def test_loads_stay_behind_the_wait(name, params, body):
    waits = re.findall(r"pdl_wait\(([^)]*)\)", body)
    assert len(waits) == 1
    handed = {v.strip() for v in waits[0].split(",") if v.strip()}
    # Pointers that the compiler may take for read-only memory.
    for p in re.findall(r"const\s+[\w:<> ]+\*\s*__restrict__\s*(\w+)", params):
        assert p in STATIC or p in POPULATIONS or p in handed, p
    # Loads that depend on their address alone need an index or pointer from the wait.
    after = body[body.index("pdl_wait("):]
    if re.search(r"kIndexed|\bChildRecord<S>::|\bld_rec\(", after):
        assert handed, "loads free to be scheduled without an index from the wait"
    assert "__ldg(" not in after


def test_population_and_record_loads_are_ordered():
    s = code(CSRC / "d3q19.cuh")
    assert re.search(r"template <int R = kOrdered>\s*__device__ __forceinline__ static float ld\(", s)
    assert re.search(r"template <int R = kOrdered>\s*__device__ __forceinline__ static float ld_dev\(", s)
    for m in re.finditer(r"asm( volatile)?\(\"ld\.global(\.nc)?", s):
        line = s[s.rfind("\n", 0, m.start()) + 1:m.start()]
        if "kOrdered" in line:
            assert m.group(1) and not m.group(2)
        elif "kIndexed" in line:
            assert not m.group(2)
    assert "__ldg(" not in code(CSRC / "child_record.cuh")
    # The read-only path past the wait: only the restriction's own cells, which
    # the coarse collide wrote launches ago.
    uses = [(p.name, m) for p in CSRC.glob("*.cu*") for m in re.findall(r"kEarlier>\((\w+)", code(p))]
    assert uses == [("refine_kernels.cu", "fc")]
