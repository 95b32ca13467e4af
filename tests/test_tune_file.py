"""Recorded configuration choices survive a file, the first entry of a box included (no GPU needed)."""
import ladderdga_b200 as L


def test_first_entries_are_written(tmp_path):
    src, out = tmp_path / "in.txt", tmp_path / "out.txt"
    want = ["bse 20 2 warp:1", "bse 30 2 warp:1", "bse 40 1 lu8:6", "bse 60 2 lu16:2"]
    src.write_text("\n".join(want) + "\n")
    L.tune_reset()
    try:
        L.tune_load(src)
        L.tune_save(out)
        assert sorted(l for l in out.read_text().splitlines() if not l.startswith("#")) == want
    finally:
        L.tune_reset()
