"""build() makes the secondary oracle only from a tree that holds the sources: an
empty reference mount is no tree."""

import __graft_entry__ as g


def test_empty_mount_is_no_tree(tmp_path, monkeypatch):
    assert not g._has_sources(str(tmp_path))
    (tmp_path / "sporco_cuda" / "src").mkdir(parents=True)
    assert g._has_sources(str(tmp_path))
    monkeypatch.delenv("SPORCO_REFERENCE_DIR", raising=False)
    monkeypatch.setattr(g, "_has_sources", lambda d: False)
    assert g._reference_dir() is None
