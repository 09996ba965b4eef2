"""Every call of the CUDA runtime in the host extension has its result looked
at: wrapped in C10_CUDA_CHECK, compared, or clearing an error already seen."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "universal-beta-splatting_gb300", "csrc", "host", "native.cpp")


def test_cuda_results_are_checked():
    with open(SRC) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    calls = [m for m in re.finditer(r"\bcuda[A-Z]\w*\s*\(", text)]
    assert calls
    for m in calls:
        name = m.group(0).rstrip("( ")
        if name == "cudaGetLastError":
            continue
        # the statement so far: a bare call starts it
        before = re.split(r"[;{}]", text[:m.start()])[-1].strip()
        assert before, "%s: result dropped" % name
        assert "C10_CUDA_CHECK(" in before or before.startswith("if (") and "!=" in text[
            m.start():m.start() + 300], "%s: result dropped (%r)" % (name, before)
