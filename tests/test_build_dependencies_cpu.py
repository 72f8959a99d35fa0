"""What the build recompiles (CPU, nvcc replaced by a recorder): every translation unit after an edit to any header that the
sources include, nothing when nothing changed."""
import os
import re

from cuequivariance_b200 import build as B


def test_every_included_header_is_a_dependency():
    known = {p.resolve() for p in B.headers()}
    for src in list(B.CSRC.rglob("*.cu")) + list(B.CSRC.rglob("*.cuh")) + list(B.CSRC.rglob("*.h")):
        for name in re.findall(r'^\s*#\s*include\s+"([^"]+)"', src.read_text(), flags=re.M):
            assert (src.parent / name).resolve() in known, (src.name, name)


def test_an_edited_header_rebuilds_every_object(monkeypatch, tmp_path):
    root = tmp_path / "repo"
    csrc, inc = root / "pkg" / "csrc", root / "include"
    csrc.mkdir(parents=True), inc.mkdir()
    for n in ("a.cu", "b.cu", "shared.h", "dev.cuh"):
        (csrc / n).write_text("")
    (inc / "api.h").write_text("")
    ran = []

    class _Run:
        returncode, stdout = 0, ""

        def __init__(self, cmd, **kw):
            out = cmd[cmd.index("-o") + 1]
            ran.append(os.path.basename(out))
            open(out, "w").close()

        def communicate(self):
            return "", None

    monkeypatch.setattr(B, "ROOT", root), monkeypatch.setattr(B, "PKG", root / "pkg"), monkeypatch.setattr(B, "CSRC", csrc)
    monkeypatch.setattr(B, "LIB", root / "pkg" / "lib.so"), monkeypatch.setattr(B, "generate", lambda: None)
    monkeypatch.setattr(B.subprocess, "Popen", _Run), monkeypatch.setattr(B.subprocess, "run", _Run)
    B.build()
    assert sorted(ran) == ["a.o", "b.o", "lib.so"]
    ran.clear()
    B.build()
    assert ran == []
    for name in (csrc / "shared.h", csrc / "dev.cuh", inc / "api.h"):
        newer = max(p.stat().st_mtime for p in root.rglob("*")) + 10
        os.utime(name, (newer, newer))
        assert B._stale()
        ran.clear()
        B.build()
        assert sorted(ran) == ["a.o", "b.o", "lib.so"], name
        for out in list((root / "pkg" / "build").glob("*.o")) + [B.LIB]:
            os.utime(out, (newer + 1, newer + 1))
