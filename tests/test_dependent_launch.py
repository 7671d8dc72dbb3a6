"""Kernels that may start before the stream's previous kernel has ended (programmatic dependent
launch) read what it wrote only through pointers that the wait has given back: otherwise the compiler
may move a load that it takes for read-only above the wait.  Nothing here runs: the rule is checked in
the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "akuaengine_gb300",
                    "csrc")
WAIT = "wait_for_previous("


def _sources():
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            out[os.path.basename(path)] = re.sub(r"//[^\n]*", "", f.read())
    return out


def _balanced(text, at, pair):
    """text[at] opens a bracket: the index just past its partner."""
    depth = 0
    for k in range(at, len(text)):
        depth += text[k] == pair[0]
        depth -= text[k] == pair[1]
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced source")


def _kernels():
    """(file, name, parameters, body) of every kernel."""
    found = []
    for name, text in _sources().items():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__)?", text):
            at = m.end()
            if text[at] == "(":  # __launch_bounds__(...)
                at = _balanced(text, at, "()")
            k = re.compile(r"\s*(\w+)\s*\(").match(text, at)
            end = _balanced(text, k.end() - 1, "()")
            body = text.index("{", end)
            found.append((name, k.group(1), text[k.end():end - 1],
                          text[body:_balanced(text, body, "{}")]))
    return found


def test_one_wait():
    uses = {f: t.count("griddepcontrol.wait") for f, t in _sources().items()}
    assert {f: n for f, n in uses.items() if n} == {"dependent_launch.cuh": 1}


# What the kernel before it in a step or a sort may write of a kernel's inputs.  All that kernels before
# that one wrote is complete when a kernel starts.
PREVIOUS = {
    "k_table_build": {"r2i"},                           # k_gather
    "k_density_lambda": {"ps"},                         # k_delta_correct
    "k_delta_correct": {"lam", "psl", "nbr4", "cnt"},   # k_search, k_mlp_forward, k_density_lambda
    "k_delta_final": {"lam", "psl", "nbr4", "cnt"},
    "k_vorticity": {"x4", "v4", "xv8"},                 # k_delta_final
    "k_confine": {"om4", "xw4"},                        # k_vorticity
    "k_xsph": {"xv8"},                                  # k_confine
    "k_export": {"v4"},                                 # k_xsph
    "upsweep": {"keys"},                                # the last pass
    "scan_tiles": {"counts"},                           # upsweep
    "downsweep": {"counts", "totals"},                  # upsweep, scan_tiles
    "cluster_pass": {"keys_in", "vals_in"},             # the last pass
    "k_mlp_adam": {"params", "grad", "m", "v"},
}


def _waiting():
    return [k for k in _kernels() if WAIT in k[3]]


def test_waiting_kernels_are_found():
    names = {k[1] for k in _waiting()}
    assert set(PREVIOUS) | {"k_mlp_forward", "k_mlp_grad", "k_splat_large", "k_splat_resolve"} == names


def test_kernels_set_up_early_wait():
    """The kernels of a step that are launched with the attribute (step_kernel)."""
    names = {k[1] for k in _waiting()}
    early = set()
    for text in _sources().values():
        early |= set(re.findall(r"\bstep_kernel\(s, st, (?:akua::)?(k_\w+)", text))
        assert not re.search(r"\bstep_kernel\(s, st, (?!(?:akua::)?k_)", text)
    assert {"k_table_build", "k_density_lambda", "k_export"} <= early <= names, early - names


@pytest.mark.parametrize("kernel", _waiting(), ids=lambda k: k[1])
def test_inputs_come_out_of_the_wait(kernel):
    """Kernels that may follow anything (the network's, the renderer's) pass every input."""
    _, name, params, body = kernel
    at = body.index(WAIT) + len(WAIT) - 1
    given = {a.strip() for a in body[at + 1:_balanced(body, at, "()") - 1].split(",")}
    inputs = set()
    for p in re.sub(r"__\w+__", "", params).split(","):
        m = re.match(r"\s*const\s+[\w ]*?\s*\*\s*(\w+)\s*$", p)
        if m:
            inputs.add(m.group(1))
    need = PREVIOUS.get(name, inputs)
    assert need <= given, "%s reads %s past its wait" % (name, sorted(need - given))
    before = re.sub(r'"[^"]*"', "", body[:at])
    early = [p for p in given if re.search(r"\b%s\b" % p, before)]
    assert not early, "%s uses %s before its wait" % (name, early)
    assert not [p for p in given if re.search(r"__ldg\(\s*&?%s\b" % p, body)]


def test_no_read_only_loads():
    """No .nc load, no load that the compiler takes for a pure function of its address, and no __ldg in
    the helpers that several waiting kernels share."""
    for name, text in _sources().items():
        for m in re.finditer(r"\basm(\s+volatile)?\s*\(\s*\"(ld[\w.:]*)", text):
            assert m.group(1) and ".nc" not in m.group(2), "%s: %s" % (name, m.group(2))
        if name in ("pbf_pairs.cuh", "radix_sort.cuh", "mlp.cuh", "splat.cu"):
            assert "__ldg(" not in text, name
