"""The in-tree build with a compiler that stands in for nvcc (CPU)."""
import os
import stat
import threading
from pathlib import Path

FAKE = """#!/usr/bin/env python3
import sys, time
out, args = sys.argv[sys.argv.index("-o") + 1], sys.argv[1:]
if "-c" in args:
    open(out, "w").write("{name} ")
    time.sleep({wait})
else:
    time.sleep({wait})
    open(out, "w").write("".join(open(a).read() for a in args if a.endswith(".o") and a != out))
"""


def test_builds_at_once_do_not_share_objects(tmp_path, monkeypatch):
    """Two builds overlap, the second starting while the first still compiles: each links its own two
    objects, the library is one of them whole, and nothing else is left beside it."""
    from axtb_b200 import build as B

    out = tmp_path / "libaxtb_gpu.so"
    monkeypatch.setattr(B, "OUT", out)
    fakes = []
    for name, wait in (("first", 0.6), ("second", 0.3)):
        path = tmp_path / name
        path.write_text(FAKE.format(name=name, wait=wait))
        path.chmod(path.stat().st_mode | stat.S_IXUSR)
        fakes.append(str(path))
    which = threading.local()
    monkeypatch.setattr(B, "nvcc", lambda: which.path)
    errors, seen = [], []

    def run(path, delay):
        which.path = path
        threading.Event().wait(delay)
        try:
            B.build(force=True)
            seen.append(out.read_text())
        except Exception as e:  # reported below
            errors.append(e)

    threads = [threading.Thread(target=run, args=(p, d)) for p, d in zip(fakes, (0.0, 0.3))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert set(seen) <= {"first first ", "second second "} and len(seen) == 2
    assert sorted(os.listdir(tmp_path)) == ["first", "libaxtb_gpu.so", "second"]
    assert isinstance(B.OUT, Path)


def test_documented_command_is_the_build(engine):
    """The nvcc command that the integration guide gives has the build's flags and sources."""
    from axtb_b200 import build as B

    root = Path(B.__file__).resolve().parent.parent
    words = next(line for line in (root / "INTEGRATION.md").read_text().splitlines() if line.startswith("`nvcc ")).strip("`)").split()
    assert words[0] == "nvcc" and set(B.FLAGS) <= set(words)
    assert [w for w in words if w.endswith(".cu")] == [str(p.relative_to(root)) for p in (B.SRC, B.TRD)]
    assert words[words.index("-o") + 1] == str(B.OUT.relative_to(root))
