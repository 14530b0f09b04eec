"""The autotuner's cache holds for the build of the library that was timed: another build's
kernels are timed anew, and the first build's choice is kept beside it."""
import json

import pytest
import torch

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import batched as B
from reduced_mpm_stress_training_gb300 import scenarios as S


@pytest.fixture
def timed(monkeypatch, tmp_path):
    calls = []

    def time_chunk_size(scenes, chunk, device, steps=8):
        calls.append(chunk)
        return timed.seconds[chunk]

    timed.seconds = {64: 1.0, 128: 2.0}
    monkeypatch.setenv("MPM_GB300_CACHE", str(tmp_path / "cache"))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "a GPU")
    monkeypatch.setattr(B, "time_chunk_size", time_chunk_size)
    library = tmp_path / "libmpm_gb300.so"
    library.write_bytes(b"first build")
    monkeypatch.setattr(A, "lib_path", lambda: str(library))
    timed.calls, timed.library, timed.cache = calls, library, tmp_path / "cache" / "autotune.json"
    return timed


def _tune():
    return B.autotune([S.small_column(100, 16), S.small_column(200, 16)], candidates=(64, 128))


def test_a_choice_is_kept_for_its_build(timed):
    assert _tune() == 64 and timed.calls == [64, 128]
    assert _tune() == 64 and timed.calls == [64, 128]  # cached
    timed.library.write_bytes(b"second build")
    timed.seconds = {64: 2.0, 128: 1.0}
    assert _tune() == 128 and timed.calls == [64, 128] * 2  # timed anew
    assert _tune() == 128 and timed.calls == [64, 128] * 2
    timed.library.write_bytes(b"first build")
    assert _tune() == 64 and timed.calls == [64, 128] * 2
    assert len(json.loads(timed.cache.read_text())) == 2


def test_other_workloads_keep_their_own_choice(timed):
    _tune()
    assert B.autotune([S.small_column(300, 16)], candidates=(64, 128)) == 64
    assert len(json.loads(timed.cache.read_text())) == 2
