"""The autotuner's cache holds timings of this build's kernels and of the kernels an instance runs: entries of other
builds and of other variants are not used (no GPU: the timing itself is replaced)."""
import pytest

torch = pytest.importorskip("torch")

import cdd
from cdd import autotune


@pytest.fixture
def tuner(tmp_path, monkeypatch):
    monkeypatch.setenv("CDD_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "GPU")
    monkeypatch.setattr(autotune, "library_tag", lambda: "build1")
    calls = []

    def tune(inst, precision, **kw):
        calls.append(inst)
        return {"stencil_planes": len(calls)}, 1.0, 2.0, []

    monkeypatch.setattr(autotune, "tune", tune)
    return calls, monkeypatch


def test_entries_of_other_builds_are_not_used(tuner):
    calls, monkeypatch = tuner
    inst = cdd.Instance((32, 32, 32))
    old = autotune.cache_key("GPU", "f32", inst.shape)
    other = autotune.cache_key("GPU", "f32", (32, 32, 64))
    autotune.save_cache({old: {"tuning": {"stencil_planes": 99}}, other: {"tuning": {"stencil_planes": 98}}})
    assert autotune.best(inst, "f32") == {"stencil_planes": 1}
    assert autotune.best(inst, "f32") == {"stencil_planes": 1} and len(calls) == 1
    monkeypatch.setattr(autotune, "library_tag", lambda: "build2")
    assert autotune.best(inst, "f32") == {"stencil_planes": 2} and len(calls) == 2
    assert len(autotune.load_cache()) == 2 and other in autotune.load_cache()


def test_variants_have_entries_of_their_own(tuner):
    calls, _ = tuner
    kinds = [{}, {"glide_only": True}, {"vacancy": (0.4, 0.7, 0.02)}, {"Lambda": 0.1}]
    for _ in range(2):
        for kw in kinds:
            autotune.best(cdd.Instance((32, 32, 32), **kw), "f64")
    assert len(calls) == len(kinds) == len(autotune.load_cache())


def test_library_tag_is_a_digest_of_the_library():
    assert len(autotune.library_tag()) == 16
