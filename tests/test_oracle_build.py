"""The oracle's build without the reference's sources."""


def test_an_empty_reference_folder_counts_as_none(oracle_mod, monkeypatch, tmp_path):
    monkeypatch.setattr(oracle_mod, "REFERENCE_DIR", str(tmp_path))
    monkeypatch.setattr(oracle_mod, "REF_SO", str(tmp_path / "ref.so"))
    oracle_mod.build()
    assert list(tmp_path.iterdir()) == []


def test_the_reference_is_absent_where_its_sources_are(oracle_mod, monkeypatch, tmp_path):
    monkeypatch.setenv("IDG_REFERENCE_DIR", str(tmp_path))
    assert oracle_mod._reference_dir() == ""
    (tmp_path / "gridding" / "src").mkdir(parents=True)
    assert oracle_mod._reference_dir() == str(tmp_path)
