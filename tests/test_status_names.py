"""Every code that a wait of a kernel can leave behind has a name, and its own."""
import glob
import os
import re

from helpers import ROOT


def _codes():
    got = {}
    for path in glob.glob(os.path.join(ROOT, "sparse_mla_sm120_b200", "csrc", "*.cu")):
        with open(path) as f:
            text = f.read()
        for enum in re.findall(r"enum \{([^}]*)\}", text):
            got.update((name, int(code)) for name, code in re.findall(r"\b(W[A-Z]?_\w+) = (\d+)", enum))
        # a code stands at its wait by name only
        assert not re.search(r"mbar_wait\w*\(.*, abort_\w+, \d+\)", text), path
    return got


def test_every_code_has_a_name_of_its_own():
    from sparse_mla_sm120_b200 import _lib
    name = {k: _lib.load().smla_status_string(v).decode() for k, v in _codes().items()}
    assert len(name) >= 48 and "unknown" not in name.values() and len(set(name.values())) == len(name)


def test_names_say_which_wait():
    from sparse_mla_sm120_b200 import _lib
    for wait, code in _codes().items():
        if wait.startswith(("WL_", "WD_")):
            assert wait[3:].lower().replace("_", "") in _lib.load().smla_status_string(code).decode().replace("_", "").replace(" ", ""), wait
