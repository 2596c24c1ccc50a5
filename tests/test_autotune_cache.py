"""The autotuner's cache: an entry of another version of the tuned kernels is
not taken over (no GPU: a scene that only answers what the key asks)."""
import json

import pytest

from cudaraytracer_b200 import autotune


class FakeScene:
    class ctx:
        device = 0

    def __init__(self):
        self.set = {}

    def info(self):
        return {"num_triangles": 36}

    def render_params(self):
        return {"width": 64, "height": 48, "max_bounces": 5}

    def set_render_params(self, **kw):
        self.set.update(kw)


def test_entries_of_other_versions_are_tuned_again(tmp_path, monkeypatch):
    import torch

    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d: "GPU")
    entry = {"paths_per_pass": 4096, "stage_block": 256, "stage_traversal": 2}
    cache, sc = tmp_path / "tune.json", FakeScene()
    key = autotune.cache_key(sc, 3)
    cache.write_text(json.dumps({key: entry}))
    got = autotune.autotune_paths_per_pass(sc, [None] * 3, cache_path=str(cache))
    assert got["cached"] and sc.set == entry
    # the key of before there was a version, and an older version's
    for old in ("GPU|tris2^5|64x48x3|bounces5", key.replace(f"v{autotune.VERSION}|", "v1|")):
        assert old != key
        cache.write_text(json.dumps({old: entry}))
        monkeypatch.setattr(torch, "zeros", lambda *a, **k: (_ for _ in ()).throw(RuntimeError("tunes")))
        with pytest.raises(RuntimeError, match="tunes"):
            autotune.autotune_paths_per_pass(sc, [None] * 3, cache_path=str(cache))
