"""Kernels launched with programmatic serialisation (launch_chained) are resident
before the kernel that writes their input has ended. CUDA lets the compiler read
`const __restrict__` pointers, and __ldg reads, through the read-only path,
whose contract is that the memory does not change while the kernel is resident,
and it may move such reads above the wait. So what a kernel of a chain writes
must be read through plain pointers. Checked in the sources: every kernel that
calls chain_wait, the functions it hands those pointers to, and the structs
that carry the displacement words."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mars_md_b200", "csrc")
# What chained kernels write, by the names of the parameters that carry it.
WRITTEN = {"pos", "from", "mom", "fe", "fs", "force", "sorted_pos", "ref", "clear", "clear_a", "clear_b",
           "lam", "mu", "mu_sorted", "tan", "tan_sorted", "moved", "d2max", "d2sys", "step_ptr"}


def _sources():
    return {os.path.basename(f): open(f).read() for f in sorted(glob.glob(CSRC + "/*.cu*"))}


def _functions(text):
    """(name, parameter list, body) of each device function and kernel."""
    for m in re.finditer(r"(?:__global__|__device__)[^;{]*?(\w+)\(((?:[^()]|\([^()]*\))*)\)\s*(?:const\s*)?\{", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), m.group(2), text[m.end():i]


def _restricted(params):
    return [m.group(1) for m in re.finditer(r"__restrict__\s+(\w+)", params)]


def _chained():
    return [(f, name, params, body) for f, text in _sources().items()
            for name, params, body in _functions(text) if "chain_wait()" in body and name != "chain_wait"]


def test_every_chained_launch_is_covered():
    names = {name for _, name, _, _ in _chained()}
    assert {"pack_kernel", "batch_pack_kernel", "fast_pair_kernel", "pair_force_kernel",
            "bond_angle_kernel", "bd_gather_kernel", "baoab_kernel", "bd_systems_kernel",
            "adj_mu_kernel", "adj_pair_kernel", "adj_bond_angle_kernel", "adj_combine_kernel"} <= names


@pytest.mark.parametrize("file,name,params,body", _chained(), ids=lambda v: v if len(v) < 40 else "")
def test_chained_kernels_read_what_a_chain_writes_plainly(file, name, params, body):
    assert not set(_restricted(params)) & WRITTEN, (file, name)
    for m in re.finditer(r"__ldg\(\s*&?\s*([\w.]+)", body):
        assert m.group(1).split(".")[-1] not in WRITTEN, (file, name, m.group(0))


@pytest.mark.parametrize("name", ["bond_term", "angle_term", "adj_bonds", "adj_angle"])
def test_their_device_functions_do_too(name):
    found = [p for text in _sources().values() for n, p, _ in _functions(text) if n == name]
    assert found and not any(set(_restricted(p)) & WRITTEN for p in found)


def test_displacement_words_are_read_plainly():
    text = _sources()["mb2_forces.cu"]
    for struct in ("OneBox", "SystemBoxes"):
        body = text[text.index("struct " + struct + " {"):]
        body = body[:body.index("\n};")]
        assert not set(_restricted(body)) & WRITTEN and "__ldg" not in body
