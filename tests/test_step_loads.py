"""Loads of the step kernels (source check, CPU).

The step kernels launch with programmatic stream serialization: they start
while the pass before them still writes the state they read.  Loads through the
read-only path (__ldg, or const __restrict__ pointers) are defined only for
memory that nobody writes during the kernel's lifetime, so in these kernels
they are for the geometry masks and the batch's descriptors alone."""
import os
import re

from helpers import REPO

CSRC = os.path.join(REPO, "fvm-airidynamic-simulator_b200", "csrc")


def _source(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)


def _bodies(src):
    """(name, text) of every function, split at the lines that start one."""
    src = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", src)
    parts = re.split(r"^(?=(?:template|__global__|__device__|static|cudaError_t|size_t|int)\b)", src, flags=re.M)
    out, head = [], ""
    for part in parts:
        if part.startswith("template") and "(" not in part:
            head = part
            continue
        m = re.search(r"(\w+)\(", part)
        if m:
            out.append((m.group(1), head + part))
        head = ""
    return out


def _arguments(text):
    """Arguments of every __ldg call."""
    out = []
    for m in re.finditer(r"__ldg\(", text):
        k, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        out.append(text[m.end():k - 1])
    return out


# passes of the set-up path, launched plainly
PLAIN = {"k_bc_phase1", "k_cfl_state"}


def test_step_kernels_read_states_with_ordinary_loads():
    src = _source("fvm_step.cu")
    bodies = _bodies(src)
    names = {n for n, _ in bodies}
    assert PLAIN | {"flat_tile", "k_stage", "k_stage_flat", "k_stage_flat_batch", "k_viscous", "k_ghost"} <= names, names
    for name in PLAIN:  # and stay launched plainly
        assert re.search(name + r"<<<", src) and not re.search(r"launch_step_kernel\([^;]*\b" + name, src), name
    for name, text in bodies:
        if name in PLAIN:
            continue
        for arg in _arguments(text):
            assert re.search(r"\bmask\b|\bmcol\b", arg), (name, arg)
        for m in re.finditer(r"const\s+(\w+)\s*\*\s*__restrict__", text):
            assert m.group(1) in ("BatchInst", "TileDesc", "GhostChunk"), (name, m.group(0))
        assert "load4(" not in text, name  # fvm_quads.cuh: read-only loads
