"""The build entry point without H2Pack's sources: the CUDA engine builds and loads by itself,
and a missing GPU build of H2Pack is said, not raised."""
import __graft_entry__ as entry


def test_build_without_h2pack_sources(monkeypatch, tmp_path, capsys):
    made = []
    monkeypatch.setattr(entry, "REF_SRC", str(tmp_path / "none"))
    monkeypatch.setattr(entry, "_make", lambda path, extra=(): made.append((path, [e.rsplit("/", 1)[-1] for e in extra])))
    monkeypatch.setattr(entry, "_has_dropin", lambda: False)
    entry.build()
    assert made == [("h2pack_b200", ["libh2gpu.so"])]
    assert "libH2Pack_gpu.so" in capsys.readouterr().out


def test_reference_arm_says_when_the_library_is_not_there(monkeypatch, capsys):
    import json
    import sys
    import bench
    from oracle import oracle
    monkeypatch.setattr(oracle, "have_ref", lambda: False)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1"])
    bench.main()
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "not built" in line["unavailable"]
