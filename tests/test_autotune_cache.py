"""The launch-shape cache: an entry is re-applied with the library build that it
was timed with, and timed again with any other (a stub stands for the library)."""
import json

import pytest

from adc_ottawa_gb300 import autotune


class _Lib:
    def __init__(self):
        self.tuned, self.applied = 0, []

    def adcgpu_sigma_autotune(self, h, m, chunk, mc, ms):
        self.tuned += 1
        chunk._obj.value, mc._obj.value, ms._obj.value = 64, 2, 1.5
        return 0

    def adcgpu_sigma_set_shape(self, h, chunk, mc64, mc32):
        self.applied.append((chunk, mc64, mc32))
        return 0


class _Context:
    nocc, nvirt, _h = 10, 110, None

    def _check(self, st, what):
        assert st == 0, what


@pytest.fixture
def stub(monkeypatch):
    s = _Lib()
    monkeypatch.setattr(autotune, "lib", lambda: s)
    monkeypatch.setattr(autotune, "_build", lambda: "this", raising=False)
    return s


# 16: the per-warp kernels, which the entry of an older build may ask for where
# this one has faster ones
@pytest.mark.parametrize("entry", [{"chunk": 16, "mc": 18, "ms": 9.7},
                                   {"chunk": 16, "mc": 18, "ms": 9.7, "build": "other"}])
def test_entry_of_another_build_is_timed_again(stub, tmp_path, entry):
    cache = tmp_path / "tune.json"
    cache.write_text(json.dumps({"no10-nv110-p0-m10": entry}))
    r = autotune.tune(_Context(), 10, 0, cache=str(cache))
    assert not r["cached"] and stub.tuned == 1 and not stub.applied
    r = autotune.tune(_Context(), 10, 0, cache=str(cache))
    assert r["cached"] and stub.tuned == 1 and stub.applied == [(64, 2, 4)]
    assert autotune.tune(_Context(), 10, 0, cache=str(cache), force=True)["cached"] is False


def test_build_follows_the_library(monkeypatch, tmp_path):
    so = tmp_path / "lib.so"
    monkeypatch.setattr(autotune, "LIB_PATH", str(so))
    seen = set()
    for text in (b"one", b"two"):
        so.write_bytes(text)
        autotune._build.cache_clear()
        seen.add(autotune._build())
    autotune._build.cache_clear()
    assert len(seen) == 2
