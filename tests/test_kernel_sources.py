"""Rules that the CUDA sources have to keep and that no run can show: checked on
the text of the kernels."""
import os
import re

import gpe_b200

CSRC = os.path.join(os.path.dirname(gpe_b200.__file__), "csrc")
DEF = re.compile(r"\b(\w+)\s*\(([^;{}]*?)\)\s*\{", re.S)
# per-axis weights, uploaded when the context is created
CONSTANT_TABLES = {"wx", "wy", "wz"}


def functions():
    """name -> (parameter list, body) of every device function and kernel."""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, f)) as h:
            s = re.sub(r"//[^\n]*", "", h.read())
        for m in re.finditer(r"__(?:global|device)__\s", s):
            # past __launch_bounds__(...), whose parentheses are not the parameters
            at = m.end()
            lb = re.match(r"(?:__forceinline__\s+|inline\s+)?[\w:<>,*&\s]*?__launch_bounds__\(", s[at:])
            if lb:
                at += lb.end()
                at = s.index(")", at) + 1
                while s[at - 1] != ")" or s[m.end():at].count("(") != s[m.end():at].count(")"):
                    at = s.index(")", at) + 1
            d = DEF.search(s, at)
            semi = s.find(";", at)
            if not d or (semi >= 0 and semi < d.start()):
                continue
            depth, end = 1, d.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(s[end], 0)
                end += 1
            out.setdefault(d.group(1), []).append((d.group(2), s[d.end():end]))
    return out


def reached(fns, name, seen):
    if name in seen:
        return seen
    seen.add(name)
    for _, body in fns[name]:
        for word in set(re.findall(r"\b\w+\b(?=\s*(?:<[^;(){}]*>)?\s*\()", body)):
            if word in fns:
                reached(fns, word, seen)
    return seen


def test_overlapped_kernels_promise_nothing_about_memory_in_flight():
    """A kernel that waits for the one before it (after_previous) is running
    while that one still writes: a __restrict__ pointer to what it writes would
    let the compiler load before the wait."""
    fns = functions()
    kernels = {n for n in fns if n.endswith("_kernel") or "_kernel_" in n}
    assert len(kernels) > 30
    overlapped = [k for k in kernels if "after_previous" in reached(fns, k, set())]
    assert {"finalize_kernel", "ghosts_norm_kernel", "rescale_to_kernel", "pack_input_kernel",
            "loss_kernel", "grad_finalize_kernel", "conv_fwd_kernel", "stage_kernel",
            "pair_kernel"} <= set(overlapped)
    bad = set()
    for k in overlapped:
        for f in reached(fns, k, set()):
            for params, _ in fns[f]:
                for p in re.findall(r"__restrict__\s+(\w+)", params):
                    if p not in CONSTANT_TABLES:
                        bad.add((k, f, p))
    assert not bad, sorted(bad)


def test_every_launch_asks_the_rule_for_overlap():
    """Launches overlap where the context's rule lets them (not while each is
    timed by itself, for one): none says so by itself."""
    calls = []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            with open(os.path.join(CSRC, f)) as h:
                calls += re.findall(r"launch_overlapped\(\s*([^,]+),", h.read())
    assert len(calls) >= 15
    assert set(calls) <= {"overlap(c)", "ov", "v.overlap"}, sorted(set(calls))


def test_members_of_a_batch_lie_along_the_x_of_a_grid():
    """A grid has 65535 blocks along y and z: a launch with one per member there
    would refuse batches that the others take."""
    for name, defs in functions().items():
        for _, body in defs:
            assert "blockIdx.y" not in body and "blockIdx.z" not in body, name
