"""The autotuner's cache across libraries: an entry without the table version in
its key, as a library wrote it whose tiling ids meant other kernels, is not
applied; the entry written now is, and a network of another depth has its own."""
import pytest

pytestmark = pytest.mark.gpu


def test_entries_of_another_tiling_table(nmg, synth, tmp_path, monkeypatch):
    import torch
    path = tmp_path / "tune.txt"
    monkeypatch.setenv("NMG_TUNE_CACHE", str(path))
    n = 20000
    q = synth.wavefront(n, seed=3)
    a = [torch.from_numpy(q[k]).cuda() for k in ("pos", "wo", "normal", "rough", "u4")]
    f = nmg.GuidingField(nmg.config(1, path=1), max_queries=n)
    deep = nmg.GuidingField(nmg.config(1, path=1, hidden_layers=7), max_queries=n)
    try:
        f.autotune(*a, use_cache=True)
        key, value = path.read_text().split()
        old, version = key.rsplit("|t", 1)
        assert int(version) >= 2
        assert "|h3|" in old
        path.write_text("%s 10\n" % old.replace("|h3|", "|"))  # an older library's key and winner
        f.autotune(*a, use_cache=True)
        assert path.read_text().split()[2] == key  # timed again, and stored under today's key
        path.write_text("%s 10\n" % key)
        assert f.autotune(*a, use_cache=True) == 10 and f.query_tiling == 10
        deep.autotune(*a, use_cache=True)
        assert len(path.read_text().splitlines()) == 2
    finally:
        f.close()
        deep.close()
