"""The autotuner's cache on disk, without a GPU: what an earlier library chose
among fewer launch shapes does not keep this one from its new ones."""
import json

import pytest


@pytest.mark.parametrize("timed,applies", [((26, 41), True), ((25, 40), False), ((0, 0), False)])
def test_a_choice_among_other_shapes_does_not_count(idg, monkeypatch, tmp_path, timed, applies):
    from idg_gb300 import tuning
    from idg_gb300.ops import GridSpec

    spec = GridSpec(1024, 32, 16, 4)
    path, chosen = tmp_path / "shapes.json", []
    monkeypatch.setenv("IDG_TUNE_CACHE", str(path))
    monkeypatch.setattr(tuning.torch.cuda, "get_device_name", lambda: "a GPU")
    monkeypatch.setattr(tuning, "num_shapes", lambda: (26, 41))
    monkeypatch.setattr(tuning, "set_shapes", lambda *a: chosen.append(a))
    entry = {"gridder": 24, "degridder": 34, "gridder_ms": [1.0] * timed[0], "degridder_ms": [1.0] * timed[1]}
    path.write_text(json.dumps({tuning._key(spec): entry}))
    assert (tuning.apply_cached(spec) == entry) == applies
    assert chosen == ([(32, 24, 34)] if applies else [])
