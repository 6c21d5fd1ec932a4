"""Saved launch shapes (host only): a table that knows of every form of the split
half-sweep is installed as it stands, one from before them only at sizes that run
by rows."""
import json


def test_saved_split_shapes(tmp_path):
    from warpflow import autotune
    split = {n: {"best": [1, 4, 1], "us": {}} for n in (80, 128, 146, 256)}
    split[64] = {"best": [4, 8, 1], "us": {}, "default": True}
    default = {n: autotune.shape("split", n) for n in split}
    p = tmp_path / "tune.json"
    try:
        autotune.save({}, p, shapes={"split": split})
        autotune.load_and_apply(p)
        for n in (80, 128, 146, 256):
            assert autotune.shape("split", n) == (1, 4, 1)
        assert autotune.shape("split", 64) == default[64]
        doc = json.loads(p.read_text())
        del doc["split_forms"]
        p.write_text(json.dumps(doc))
        autotune.load_and_apply(p)
        for n in (128, 146):
            assert autotune.shape("split", n) == (1, 4, 1)
        for n in (64, 80, 256):
            assert autotune.shape("split", n) == default[n]
    finally:
        for n in split:
            autotune.set_shape("split", n, 0, 0, 0)
