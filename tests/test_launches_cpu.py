"""Launches that may be set up before the kernel in front of them has ended (``launch`` in csrc/common.cuh): each such kernel waits first."""

import re
from pathlib import Path

import language_model_saes_b200.ops.native as native

CSRC = Path(native.__file__).parent / "csrc"


def _bodies(text: str) -> dict[str, str]:
    """Name of every ``__global__`` function -> the first statement of its body."""
    found = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__\w+__\s*(?:\([^()]*(?:\([^()]*\))?[^()]*\))?\s*)*(\w+)\(", text):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        rest = text[i:].lstrip()
        if rest.startswith("{"):
            found[m.group(1)] = rest[1:].lstrip().split(";", 1)[0]
    return found


def test_every_kernel_that_is_launched_early_waits_first():
    launched = 0
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        bodies = _bodies(text)
        names = set(re.findall(r"\blaunch\(\s*(\w+)", text)) - {"const"}  # (a function of that name)
        if "ProgrammaticStreamSerialization" in text:  # clusters, with a configuration of their own
            names |= {"enc_gemm_kernel", "fp32_gemm_kernel"} & set(bodies)
        for name in list(names):
            if name not in bodies:  # a variable: every kernel that it may stand for
                names.remove(name)
                meant = {k for given in re.findall(rf"\bauto\*?\s+{name}\s*=([^;]*);", text) for k in re.findall(r"\w+", given) if k in bodies}
                assert meant, (path.name, name)
                names |= meant
        for name in names:
            assert bodies[name] == "pdl_wait()", (path.name, name, bodies[name])
        launched += len(names)
    assert launched >= 40  # (the sources were read as they are meant to be)


def test_kernels_of_files_with_a_launch_of_their_own_wait_first():
    """Where a file sets the attribute itself, every kernel of it that is not launched plainly is taken to be launched early."""
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        if "ProgrammaticStreamSerialization" in text:
            for name, first in _bodies(text).items():
                assert first == "pdl_wait()" or re.search(rf"\blaunch_plain\(\s*{name}\b", text), (path.name, name)


def test_every_launch_is_counted():
    """Kernels are launched by the two helpers, which count; what launches by itself says so in the line before."""
    for path in sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.cpp"))):
        lines = path.read_text().split("\n")
        for before, line in zip([""] + lines, lines):
            if re.search(r"<<<|cudaLaunch(Cooperative)?Kernel(Ex|ExC)?\(|cuLaunchKernel", line):
                assert "++kernel_launches;" in before, (path.name, line)
