"""A library older than any source or header it is made of is built again."""
import os

import pytest

from opencuda_gb300 import build


@pytest.mark.parametrize("name", ["hl_device.cuh", "hl_internal.h", "hl_vote.cu"])
def test_stale_library_is_rebuilt(monkeypatch, tmp_path, name):
    csrc, out = tmp_path / "csrc", tmp_path / "_build"
    csrc.mkdir()
    out.mkdir()
    for f in build.CSRC.iterdir():
        (csrc / f.name).write_bytes(f.read_bytes())
        os.utime(csrc / f.name, (1000, 1000))
    lib = out / build.LIBNAME
    lib.write_bytes(b"")
    ran = []

    def run(cmd):
        ran.append(cmd)
        if str(lib) + ".tmp" in cmd:
            (out / (build.LIBNAME + ".tmp")).write_bytes(b"")

    monkeypatch.setattr(build, "CSRC", csrc)
    monkeypatch.setattr(build, "BUILD", out)
    monkeypatch.setattr(build, "_run", run)
    build.build_library()
    assert not ran
    later = lib.stat().st_mtime + 10
    os.utime(csrc / name, (later, later))
    build.build_library()
    assert ran
