"""The autotuner's kept choices belong to the library they were measured with
(no GPU: the device's name and the engine are stand-ins)."""
import json

import pytest
import torch

from pyheartsim_b200 import _lib, autotune


class _Instance:
    n_voxel = 70000


class _Engine:
    precision = _lib.PREC_F32

    def __init__(self):
        self.configured = None

    def slots(self):
        return [0]

    def instance(self, slot):
        return _Instance()

    def configure(self, variant, ctas_per_sm):
        self.configured = (variant, ctas_per_sm)


@pytest.fixture
def fake(monkeypatch, tmp_path):
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "GPU")
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.setenv("PHS_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    for k, content in enumerate((b"first", b"second")):
        (tmp_path / f"lib{k}.so").write_bytes(content)
    return tmp_path


def test_a_choice_is_not_taken_over_by_another_library(fake, monkeypatch):
    eng = _Engine()
    monkeypatch.setattr(_lib, "LIB_PATH", str(fake / "lib0.so"))
    key = autotune._bucket(eng)
    autotune._store_file(key, (2, 4))
    assert autotune.tune(eng)["cached"] and eng.configured == (2, 4)
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.setattr(_lib, "LIB_PATH", str(fake / "lib1.so"))
    assert autotune._bucket(eng) != key
    assert autotune._load_file().get(autotune._bucket(eng)) is None


def test_a_choice_kept_without_a_library_is_not_taken_over(fake, monkeypatch):
    eng = _Engine()
    monkeypatch.setattr(_lib, "LIB_PATH", str(fake / "lib0.so"))
    old = "|".join(("GPU", str(_lib.PREC_F32), str(1 << 16), "1"))
    with open(autotune.cache_path(), "w") as f:
        json.dump({old: [2, 4]}, f)
    assert autotune._load_file().get(autotune._bucket(eng)) is None
