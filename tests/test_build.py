"""Names of built libraries: the sources' digests are kept between calls, and a changed source or header still gives another name."""
import os


def test_a_changed_source_or_header_gives_another_library(tmp_path, monkeypatch):
    from gemmars_b200.csrc import build
    monkeypatch.setattr(build, "HERE", str(tmp_path))
    monkeypatch.setenv("GEMMARS_B200_BUILD_DIR", str(tmp_path / "built"))
    (tmp_path / "unit.cu").write_text("int a;")
    (tmp_path / "head.cuh").write_text("int b;")

    def name(*defines):
        return os.path.basename(build.library_path("unit", defines)[0])

    first, other = name(), name(("GB_X", 1))
    assert first != other and name() == first and name(("GB_X", 1)) == other
    (tmp_path / "unit.cu").write_text("int aa;")
    second = name()
    assert second != first and name() == second
    (tmp_path / "head.cuh").write_text("int bb;")
    third = name()
    assert third not in (first, second) and name() == third
    (tmp_path / "more.h").write_text("int c;")
    assert name() != third
    (tmp_path / "more.h").unlink()
    assert name() == third
    (tmp_path / "unit.cu").write_text("int a;")
    (tmp_path / "head.cuh").write_text("int b;")
    assert name() == first                        # the same sources, the same library


def test_sources_are_read_once(tmp_path, monkeypatch):
    import builtins
    from gemmars_b200.csrc import build
    monkeypatch.setattr(build, "HERE", str(tmp_path))
    monkeypatch.setenv("GEMMARS_B200_BUILD_DIR", str(tmp_path / "built"))
    (tmp_path / "unit.cu").write_text("int a;")
    (tmp_path / "head.cuh").write_text("int b;")
    build.library_path("unit")
    opened = []
    real = builtins.open
    monkeypatch.setattr(builtins, "open", lambda f, *a, **k: (opened.append(str(f)), real(f, *a, **k))[1])
    for _ in range(3):
        build.library_path("unit", (("GB_X", 1),))
    assert not [f for f in opened if f.endswith((".cu", ".cuh"))]
