"""When the native host library is built again."""

import os

import pytest

from miniworld_b200 import build


@pytest.fixture
def built(tmp_path, monkeypatch):
    """Paths of a library that has just been built."""
    for name in ("NATIVE_PATH", "NATIVE_TAG_PATH"):
        monkeypatch.setattr(build, name, tmp_path / name.lower())
    build.NATIVE_PATH.write_bytes(b"")
    build.NATIVE_TAG_PATH.write_text(build.native_tag())
    return build


def test_current_library_is_kept(built):
    assert not built.native_is_stale()


@pytest.mark.parametrize("word", ["torch", "cpython", "abi"])
def test_another_torch_interpreter_or_abi_makes_it_stale(built, word):
    assert word in built.native_tag()
    built.NATIVE_TAG_PATH.write_text(built.native_tag().replace(word, word + "x"))
    assert built.native_is_stale()


def test_a_library_of_unknown_origin_is_stale(built):
    built.NATIVE_TAG_PATH.unlink()
    assert built.native_is_stale()


@pytest.mark.parametrize("source", ["HOST_SOURCE", "HEADER", "__file__"])
def test_a_newer_source_makes_it_stale(built, source):
    newer = os.stat(getattr(built, source)).st_mtime - 10
    os.utime(built.NATIVE_PATH, (newer, newer))
    assert built.native_is_stale()


def test_no_knobs_in_the_kernels():
    """A macro that a build may set to another value than the kernels are written for (four threads per position in the backward,
    once) would compile and give wrong results: the sources have no such switches."""
    for source in sorted(build.CSRC.iterdir()):
        assert not [line for line in source.read_text().splitlines() if line.lstrip().startswith(("#if", "#ifdef", "#ifndef"))], source.name
