"""Every kernel that launch() starts waits for the one before it, as its first statement.

launch() starts kernels as programmatic dependents, whose blocks may be set up while the previous kernel still runs; a
kernel without the wait would race with it.
"""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "acc-gp_b200", "csrc")
# Started with launch_ordinary() or as a cluster: nothing runs beside them.
ORDINARY = {"k_eval_partials", "k_eval_reduce"}


def closing(text, at):
    depth = 0
    while True:
        depth += {"(": 1, ")": -1}.get(text[at], 0)
        at += 1
        if depth == 0:
            return at


def kernels():
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        for found in re.finditer(r"__global__\s+void\s+", text):
            at = found.end()
            if text.startswith("__launch_bounds__", at):
                at = closing(text, text.index("(", at))
            params = text.index("(", at)
            body = text[closing(text, params):].lstrip()
            yield name, text[at:params].strip(), body


def test_every_kernel_waits_first():
    seen = 0
    for name, kernel, body in kernels():
        assert body.startswith("{"), f"{name}: {kernel}"
        seen += 1
        if kernel not in ORDINARY:
            assert body[1:].lstrip().startswith("after_previous();"), f"{name}: {kernel}"
    assert seen > 100


def test_ordinary_kernels_are_started_that_way():
    text = open(os.path.join(CSRC, "gp_evaluate.cu")).read()
    assert not re.search(r"\blaunch\(", text)
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        assert "<<<" not in text or name == "gp_device.cuh", name
