"""Every entry of the learner that puts work on its stream selects the learner's device first:
the caller's current device may be another one.  (Read from the source: a machine with one GPU
cannot have another device current.)"""
import os
import re

from conftest import PKG_DIR


def methods(text):
    """(name, body) of the overriding methods of a class body."""
    for m in re.finditer(r"\n  [\w:<>*& ]+? (\w+)\([^{;]*\) (?:const )?override \{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


def test_learner_entries_select_their_device():
    text = open(os.path.join(PKG_DIR, "csrc", "learner.cu")).read()
    found = dict(methods(text[text.index("class Learner"):]))
    assert {"set_params", "train", "loss_grad", "infer", "warm_start", "add_solution", "set_prior"} <= set(found)
    for name, body in found.items():
        work = [body.index(w) for w in ("<<<", "st_", "v.st", "target.st") if w in body]
        if work:
            assert "cudaSetDevice(device_)" in body and body.index("cudaSetDevice(device_)") < min(work), name
