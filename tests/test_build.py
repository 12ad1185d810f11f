"""The native host module is rebuilt for another torch, interpreter or command line, not only for newer sources."""

import os


def test_host_module_is_stale_for_another_torch(tmp_path, monkeypatch):
    from reskv_b200.csrc import build

    host, source, record, torch_dir = tmp_path / "_host.so", tmp_path / "host.cpp", tmp_path / "_host.txt", tmp_path / "torch"
    torch_dir.mkdir()
    (torch_dir / "version.py").write_text("__version__ = '1'")
    for path in (source, host):
        path.write_text("")
    os.utime(source, (1, 1))
    monkeypatch.setattr(build, "HOST", host)
    monkeypatch.setattr(build, "_torch_dir", lambda: torch_dir)
    command = ["g++", "-I/torch", "host.cpp"]
    assert build._host_stale([source], command, record)  # nothing is known about the module that is there
    record.write_text(build._host_record(command))
    assert not build._host_stale([source], command, record)
    assert build._host_stale([source], [*command, "-O3"], record)
    (torch_dir / "version.py").write_text("__version__ = '2'")
    assert build._host_stale([source], command, record)
    record.write_text(build._host_record(command))
    os.utime(source)
    os.utime(host, (2, 2))
    assert build._host_stale([source], command, record)
