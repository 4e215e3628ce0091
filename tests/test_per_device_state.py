"""CPU test: a kernel's shared-memory limit belongs to a device, so no call that sets one may be remembered
for the process (the second GPU's launches would fail)."""
import os
import re

import zkutil as Z

CSRC = os.path.join(Z.ROOT, "zikkurat-algebra_b200", "csrc")


def test_no_kernel_attribute_is_set_once_a_process():
    bad = []
    for f in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, f)).read()
        for m in re.finditer(r"cudaFuncSetAttribute\s*\(", text):
            start = max(text.rfind(";", 0, m.start()), text.rfind("{", 0, m.start()), text.rfind("}", 0, m.start()))
            if re.search(r"\b(static|call_once)\b", text[start + 1:m.start()]):
                bad.append((f, text.count("\n", 0, m.start()) + 1))
    assert not bad, bad
