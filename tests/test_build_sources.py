"""The build takes the library for current only when it is newer than everything
it is compiled from: the units and every header they include, directly or not."""
import os
import re

from weldformfem_gb300 import build as B


def included(path, seen):
    """Adds the repository's headers that `path` includes, and theirs."""
    for name in re.findall(r'^\s*#include\s+"([^"]+)"', open(path).read(), re.M):
        for d in (os.path.dirname(path), B.CSRC, os.path.join(B.ROOT, "include")):
            f = os.path.normpath(os.path.join(d, name))
            if os.path.exists(f):
                if f not in seen:
                    seen.add(f)
                    included(f, seen)
                break
        else:
            raise AssertionError(f"{path}: {name} not found")
    return seen


def test_every_included_header_is_a_source():
    units = [os.path.join(B.CSRC, u) for u in B.UNITS]
    headers = set()
    for u in units:
        included(u, headers)
    assert len(headers) >= 4
    missing = headers.union(units) - {os.path.normpath(s) for s in B._sources()}
    assert not missing, sorted(missing)


def test_a_newer_header_makes_the_library_stale(tmp_path, monkeypatch):
    lib = tmp_path / "lib.so"
    lib.write_bytes(b"")
    monkeypatch.setattr(B, "LIB_PATH", str(lib))
    newest = max(os.path.getmtime(s) for s in B._sources())
    os.utime(lib, (newest + 10, newest + 10))
    assert B.up_to_date()
    times = {}
    real = os.path.getmtime
    monkeypatch.setattr(B.os.path, "getmtime", lambda p: times.get(os.path.basename(p), real(p)))
    for unit in B.UNITS:
        for header in included(os.path.join(B.CSRC, unit), set()):
            times = {os.path.basename(header): newest + 20}
            assert not B.up_to_date(), header
