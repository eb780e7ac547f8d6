"""The shared object of the reference's sources is left out where they are absent."""
import oracle as orc


def test_no_sources(tmp_path, monkeypatch):
    for d in (tmp_path / "missing", tmp_path):  # no directory, an empty one
        monkeypatch.setattr(orc, "REF_SRC", str(d))
        assert orc.build_ref() is None
