"""When the extension is compiled again."""
import os

import torch

from sparse_mla_sm120_b200 import build


def test_the_extension_follows_torch(monkeypatch, tmp_path):
    """Not as long as nothing changed; again for another torch, another command, newer sources, a lost stamp, and when asked."""
    runs = []

    def compiler(cmd, verbose):
        runs.append(cmd)
        with open(build.NATIVE_PATH, "w") as f:
            f.write("extension")
    monkeypatch.setattr(build, "NATIVE_PATH", str(tmp_path / "_smla_native.so"))
    source = tmp_path / "native.cpp"
    source.write_text("source")
    os.utime(source, (1, 1))
    monkeypatch.setattr(build, "NATIVE_SRC", str(source))
    monkeypatch.setattr(build, "_headers", lambda: [])
    monkeypatch.setattr(build, "_run", compiler)

    def built(**kw):
        before = len(runs)
        assert build.build_native(**kw) == build.NATIVE_PATH
        return len(runs) - before
    assert built() == 1 and built() == 0
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "99.0")
        assert built() == 1 and built() == 0
    assert built() == 1                            # back to this torch
    with monkeypatch.context() as m:
        m.setenv("CXX", "another-compiler")
        assert built() == 1
    assert built() == 1 and built() == 0
    os.utime(source, None)
    os.utime(build.NATIVE_PATH, (2, 2))
    assert built() == 1
    os.remove(build._stamp_path())
    assert built() == 1 and built() == 0 and built(force=True) == 1
