"""Every file that a translation unit includes from this repository makes its
object stale when it changes."""
import os
import re

import pytest


def included(path, dirs):
    for name in re.findall(r'#include "([^"]+)"', path.read_text()):
        f = next((d / name for d in dirs if (d / name).exists()), None)
        if f is not None:
            yield f
            yield from included(f, dirs)


@pytest.mark.parametrize("kind", ["cu", "cpp"])
def test_objects_depend_on_their_includes(tmp_path, monkeypatch, kind):
    import sge_build as b
    srcs = [b.CSRC / s for s in (b.CU_SRCS if kind == "cu" else b.HOST_SRCS)]
    files = sorted({f for s in srcs for f in included(s, (b.CSRC, b.INC))})
    assert files
    monkeypatch.setattr(b, "OUT", tmp_path)
    built = []
    monkeypatch.setattr(b, "_run", lambda cmd, cwd=None: built.append(cmd[-1]))
    for f in files:
        monkeypatch.setattr(b, "_stale", lambda target, deps, f=f: f in deps)
        built.clear()
        b.build_sge()
        users = {s.name for s in srcs if f in set(included(s, (b.CSRC, b.INC)))}
        objs = {os.path.basename(x) for x in built}
        for u in users:
            want = u.split(".")[0] + (".cu.o" if kind == "cu" else ".o")
            assert want in objs, f"{f.name} changes, {want} is not rebuilt"
