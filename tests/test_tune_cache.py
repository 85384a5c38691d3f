"""The autotuner's on-disk choices belong to the library they were timed on: another library
file gives other cache keys, the same one the same keys."""
import importlib


def test_key_names_the_library(cf, tmp_path):
    batch = importlib.import_module(cf.__name__ + ".batch")
    a, b = tmp_path / "a.so", tmp_path / "b.so"
    a.write_bytes(b"kernels 1")
    b.write_bytes(b"kernels 2")
    ops = cf.get_ops(221, 3, (16, 16, 16))
    key = lambda lib: batch._cache_key("dev", batch._library_signature(str(lib)), ops, (16, 16, 16), 4, 8, "fwdbwd", 50, 0, batch.KNOBS)
    assert key(a) != key(b)
    a2 = tmp_path / "c.so"
    a2.write_bytes(b"kernels 1")
    assert key(a) == key(a2)


def test_plan_key_uses_the_loaded_library(cf, tmp_path, monkeypatch):
    # the key autotune_plan looks up: a stored choice of another library is not taken
    import json

    batch = importlib.import_module(cf.__name__ + ".batch")
    N, cache = (16, 16, 16), tmp_path / "t.json"
    ops = cf.get_ops(221, 3, N)
    key = lambda lib: batch._cache_key("dev", lib, ops, N, 4, 8, "fwdbwd", 50, 0, batch.KNOBS)
    here = batch._library_signature(batch.LIB_PATH)
    cache.write_text(json.dumps({key("another"): {"tuning": {"lanes": 3}, "ms": 1.0}, key(here): {"tuning": {"lanes": 1}, "ms": 2.0}}))

    class Torch:
        class cuda:
            get_device_name = staticmethod(lambda: "dev")

    monkeypatch.setattr(batch, "_torch", lambda: Torch)
    assert cf.autotune_plan(None, ops, N=N, batch=8, cache_path=str(cache)) == ({"lanes": 1}, 2.0)
