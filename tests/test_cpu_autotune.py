"""The autotuner's cache without a GPU: whose entries it takes."""
import json

import pytest

from prc_d2z import autotune


class _Measured(Exception):
    pass


@pytest.fixture
def cache(tmp_path, monkeypatch):
    """A cache file; the device has a name, and measuring raises."""
    def measure(*a, **k):
        raise _Measured
    monkeypatch.setattr(autotune, "_device_key", lambda: "gpu|sm1")
    monkeypatch.setattr(autotune, "compute_tables", measure)
    path = tmp_path / "tune.json"
    monkeypatch.setenv("PRC_D2Z_TUNE_CACHE", str(path))
    return path


ENTRY = {"radius_batch": 8, "win_variant": 1, "ms": 1.0, "times_ms": {}}


def test_an_entry_of_an_unknown_or_other_build_is_not_taken(cache):
    # a variant that was the fastest of other kernels can be the slowest of these
    cache.write_text(json.dumps({"gpu|sm1|N=128|nr=12": ENTRY, "gpu|sm1|lib=0123456789abcdef|N=128|nr=12": ENTRY}))
    with pytest.raises(_Measured):
        autotune.tune(128, 12)


def test_an_entry_of_this_build_is(cache, tmp_path):
    import prc_d2z
    lib = autotune._library_key(prc_d2z._lib.load()._name)
    cache.write_text(json.dumps({f"gpu|sm1|lib={lib}|N=128|nr=12": ENTRY}))
    assert autotune.tuned(128, 12) == (8, 1)
    other = tmp_path / "other.so"
    other.write_bytes(b"another build")
    assert autotune._library_key(str(other)) != lib
