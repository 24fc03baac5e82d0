"""When the eager call path is built again (host code only)."""

import os
import shutil
import subprocess

import pytest

from ternel_b200 import _native, build


def test_the_test_session_has_built_it():
    assert build.binding_built_for() == build.binding_target() and not build.binding_is_stale()
    assert _native.binding() is not None


def test_another_pytorch_or_a_newer_source_makes_it_stale(monkeypatch, tmp_path):
    module, source = tmp_path / "_ternel_torch.so", tmp_path / "torch_binding.cpp"
    monkeypatch.setattr(build, "BINDING_PATH", module)
    monkeypatch.setattr(build, "BINDING_SOURCE", source)
    monkeypatch.setattr(_native, "_binding", None)
    source.write_text("")
    assert build.binding_is_stale()                                     # none there
    module.write_bytes(b"")
    assert build.binding_is_stale()                                     # one that does not say what it was built for
    stamp = module.with_suffix(".target")
    stamp.write_text(build.binding_target())
    os.utime(source, (0, 0))
    os.utime(module, (2 ** 33, 2 ** 33))
    assert not build.binding_is_stale()
    os.utime(source, (2 ** 34, 2 ** 34))
    assert build.binding_is_stale()                                     # an older module than its source
    os.utime(source, (0, 0))
    stamp.write_text("torch 1.0, cpython-39")
    assert build.binding_is_stale()
    with pytest.raises(_native.NativeLibraryMissing, match="torch 1.0"):
        _native.binding()


def test_host_functions_begin_on_a_cache_line():
    """What packs blocks loses a tenth and more where it does not."""
    if not shutil.which("nm"):
        pytest.skip("no nm")
    listed = subprocess.run(["nm", str(build.LIB_PATH)], capture_output=True, text=True, check=True).stdout.splitlines()
    codec = [line.split() for line in listed if "checked_parts" in line and "_M_run" in line or line.endswith(" T tq1_pack_blocks")]
    assert len(codec) >= 2
    for address, _, name in codec:
        assert int(address, 16) % 64 == 0, (address, name)
