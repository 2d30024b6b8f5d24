"""Stacks are found by the layer object they were made from: it is held as long as they are, so that no other layer can come to its
identity and be given them."""

import weakref
from types import SimpleNamespace


class Layer(dict):
    """A layer that can be watched."""


def test_a_built_layer_lives_until_its_stacks_are_cleared(monkeypatch):
    from tensorfold_b200 import lane_fuse

    monkeypatch.setattr(lane_fuse, "_stacks", {})
    monkeypatch.setattr(lane_fuse, "_stack", lambda layer, kind, device, group: SimpleNamespace(weight=None, added=1, sizes=()))
    model = {"config": SimpleNamespace(group=64), "layers": [Layer(k=1, v=2)]}
    lane_fuse.build(model)
    watched = weakref.ref(model["layers"][0])
    model["layers"] = [Layer(k=1, v=2)]
    assert watched() is not None and lane_fuse._project(model["layers"][0], "kv", None) is None
    model["layers"] = [watched()]
    assert lane_fuse.stats(model) == {"groups": {"zba": 0, "kv": 1, "gu": 0}, "added_bytes": 1}
    lane_fuse.clear(model)
    del model["layers"]
    assert watched() is None
