"""CPU checks of the package's host half."""
import subprocess
import sys

from conftest import REPO


def test_native_module_is_loaded_with_the_cache():
    """Not inside a process's first decode step."""
    code = ("from shard_b200 import _lib, Cache, build; build.build(); Cache(num_layers=1); assert _lib._host is not None")
    subprocess.run([sys.executable, "-c", code], cwd=REPO, check=True)


def test_a_cache_can_be_made_without_the_native_module(monkeypatch):
    from shard_b200 import Cache, _lib

    def missing():
        raise _lib.ShardError("not built")

    monkeypatch.setattr(_lib, "host", missing)
    assert Cache(num_layers=2).get_seq_length() == 0
