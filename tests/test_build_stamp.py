"""The native binding is rebuilt for another Python, another torch, other flags or other sources."""

import sys


def test_the_binding_is_stamped_with_what_it_is_made_for(lib, monkeypatch, tmp_path):
    import sysconfig

    import torch

    from tensorfold_b200 import build

    digest = build.host_digest()
    assert build.HOST_STAMP.read_text().strip() == digest == build.host_digest()
    seen = {digest}

    def differs():
        other = build.host_digest()
        assert other not in seen
        seen.add(other)

    with monkeypatch.context() as m:
        m.setattr(sys, "version", "4.0.0")
        differs()
    with monkeypatch.context() as m:
        m.setattr(sysconfig, "get_config_var", lambda name: "cpython-400-x86_64-linux-gnu")
        differs()
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "99.0")
        differs()
    with monkeypatch.context() as m:
        m.setattr(build, "HOST_FLAGS", [*build.HOST_FLAGS, "-O3"])
        differs()
    with monkeypatch.context() as m:
        for name in ("host.cpp",):
            (tmp_path / name).write_bytes((build.CSRC / name).read_bytes() + b"//")
        m.setattr(build, "CSRC", tmp_path)
        differs()
    assert build.host_digest() == digest
