"""Objects are rebuilt when a header that their source includes has changed."""
import os
import re
import shutil

import pytest

from mdynamix_gb300 import build


def _headers(path):
    """Headers beside the source that it includes, directly or not."""
    out, todo = set(), [path]
    while todo:
        for h in re.findall(r'#include "([^"]+)"', open(todo.pop()).read()):
            h = os.path.join(os.path.dirname(path), h)
            if os.path.exists(h) and h not in out:
                out.add(h)
                todo.append(h)
    return out


@pytest.mark.parametrize("source", build.SOURCES)
def test_object_follows_its_headers(source, tmp_path, monkeypatch):
    csrc = tmp_path / "csrc"
    shutil.copytree(build.CSRC, csrc)
    monkeypatch.setattr(build, "CSRC", str(csrc))
    src, obj = str(csrc / source), str(tmp_path / "o")
    open(obj, "w").close()
    now = os.path.getmtime(obj) + 10.0
    os.utime(obj, (now, now))
    assert not build._stale(obj, src)
    headers = _headers(src)
    assert headers
    for h in headers:
        old = os.path.getmtime(h)
        os.utime(h, (now + 1.0, now + 1.0))
        assert build._stale(obj, src), os.path.basename(h)
        os.utime(h, (old, old))
