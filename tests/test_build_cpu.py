"""What the build looks at before it leaves a product as it is."""
from sparsewave_b200 import build


def test_the_binding_is_rebuilt_for_another_torch(monkeypatch):
    assert build.BINDING.exists() and not build.binding_is_stale()  # built before the tests
    monkeypatch.setattr(build.metadata, "version", lambda name: "0.0.1")
    assert build.binding_is_stale()


def test_a_binding_of_unknown_origin_is_rebuilt(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "BINDING_FOR", tmp_path / "absent")
    assert build.binding_is_stale()
