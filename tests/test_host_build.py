"""When the host extension is compiled again (the compiler is not run here)."""
import importlib.util
import os

import pytest

SPEC = importlib.util.spec_from_file_location("hbsattn_b200_build", os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hbsattn_b200", "build.py"))
build = importlib.util.module_from_spec(SPEC)
SPEC.loader.exec_module(build)


@pytest.mark.parametrize("content,stale", [("[{}]", False), ("[torch 1.0, {}]", True), ("", True)])
def test_extension_of_another_torch_or_python_is_stale(content, stale, tmp_path):
    path = tmp_path / "_host.so"
    path.write_bytes(b"\x7fELF" + content.format(build.host_tag()).encode() + b"\0")
    assert build.host_is_stale(str(path)) == stale


def test_older_than_its_sources_or_missing_is_stale(tmp_path):
    path = tmp_path / "_host.so"
    assert build.host_is_stale(str(path))
    path.write_text(f"[{build.host_tag()}]")
    assert not build.host_is_stale(str(path))
    os.utime(path, (1, 1))
    assert build.host_is_stale(str(path))
