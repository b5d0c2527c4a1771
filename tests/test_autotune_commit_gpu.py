"""The autotuner's cache after a second run: for every commit size class the
reloaded window is the one the second run chose, whatever an earlier run wrote --
the short classes' own window (value 0, the cost model's choice) included."""
import pytest

pytestmark = pytest.mark.gpu


def test_retuned_commit_windows_replace_older_lines(cuda_lib, tmp_path):
    import crypto_b200 as kb
    L = kb.lib()
    lo, hi = 5, 8
    kb.kzg_srs_generate(kb.gen_scalars(2, 5, 1), 1 << hi)
    cache = tmp_path / "tune.txt"
    assert L.kb200_autotune(2, lo, hi, str(cache).encode()) == hi - lo + 1
    key = cache.read_text().split()[0]
    # an earlier run that chose 19 bits, which no class this short keeps
    cache.write_text("".join(f"{key} commit 2 {lg} 19 1.0\n" for lg in range(lo, hi + 1)))
    assert L.kb200_autotune(2, lo, hi, str(cache).encode()) == hi - lo + 1
    chosen = [L.kb200_tune_get(3, 2, lg) for lg in range(lo, hi + 1)]
    assert 19 not in chosen
    try:
        assert L.kb200_autotune_load(str(cache).encode()) > 0
        assert [L.kb200_tune_get(3, 2, lg) for lg in range(lo, hi + 1)] == chosen
    finally:
        for kind in range(4):
            for lg in range(lo, hi + 1):
                L.kb200_tune_set(kind, 2, lg, 0)
