"""The autotuner's cache key: a choice belongs to the library build that was
timed (CPU; the device name and the library file are stand-ins)."""

from types import SimpleNamespace

from jaxfun_b200 import _lib
from jaxfun_b200 import autotune as at


def _solver(**kw):
    base = {"device": "cuda:0", "N": (97, 96, 96), "padding_factor": (1.0, 1.5, 1.5),
            "nonlinear_form": "rotational", "family": "C", "precision": "fp64"}
    return SimpleNamespace(**{**base, **kw})


def test_choices_of_another_build_are_not_taken(tmp_path, monkeypatch):
    monkeypatch.setenv("JFB200_AUTOTUNE_CACHE", str(tmp_path / "cache.json"))
    monkeypatch.setattr(at.torch.cuda, "get_device_name", lambda device: "NVIDIA B200")
    keys = {}
    for name in ("first", "second"):
        lib = tmp_path / f"{name}.so"
        lib.write_bytes(name.encode())
        monkeypatch.setattr(_lib, "LIB_PATH", str(lib))
        keys[name] = at.cache_key(_solver())
        assert at.cache_key(_solver()) == keys[name]
        assert at.cache_key(_solver(precision="mixed")) != keys[name]
        if name == "first":
            at.store(keys[name], {"variant": {"pencil": 0}, "ms_per_step": 1.0, "cached": False})
    assert at.lookup(keys["first"])["variant"] == {"pencil": 0}
    assert at.lookup(keys["second"]) is None
    # a record of a build that did not name itself
    old = "NVIDIA_B200/97x96x96/pad1.5x1.5/C/rotational/fp64"
    at.store(old, {"variant": {"pencil": 0}, "ms_per_step": 1.0})
    assert at.lookup(keys["second"]) is None
