"""The oracle build without the reference's sources: a missing or an empty
checkout is no checkout, and the build goes on without it."""
from oracle import build_oracle


def test_checkout_without_sources_is_none(tmp_path, monkeypatch):
    for d in (tmp_path, tmp_path / "missing"):
        monkeypatch.setenv("WL_REFERENCE_DIR", str(d))
        assert build_oracle.reference_dir() is None
    (tmp_path / "test_compress_cpu.cc").write_text("")
    monkeypatch.setenv("WL_REFERENCE_DIR", str(tmp_path))
    assert build_oracle.reference_dir() == str(tmp_path)
