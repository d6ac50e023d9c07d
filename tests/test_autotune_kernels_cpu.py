"""The variant tuner times the kernels that there are: one at the block engine's
lengths, whatever numbers the library still accepts for it, and the Stockham
chirp-z kernels' variants."""
import pytest


@pytest.mark.parametrize("name,log2_len,kernels", [("RS_COLS", 10, 1), ("RS_COLS", 12, 1), ("RS_COLS", 6, 1),
                                                   ("CZT_ROWS", 11, 1), ("CZT_ROWS", 12, 1), ("CZT_COLS", 10, 1),
                                                   ("CZT_ROWS", 9, 4), ("CZT_COLS", 13, 2), ("RS_COLS", 14, 0)])
def test_count_is_the_number_of_kernels(name, log2_len, kernels, tmp_path):
    from xlumina_gb300 import _lib
    from xlumina_gb300.autotune import VariantTuner
    selected = []
    t = VariantTuner(path=str(tmp_path / "v.json"), device_name="dev", repeats=1,
                     select=lambda p, l, v: selected.append(v))
    pass_id = getattr(_lib, "XL_PASS_" + name)
    assert t.count(pass_id, log2_len) == kernels
    if kernels:
        t.best_variant(pass_id, log2_len, lambda: 1e-3)
        assert set(selected) == set(range(kernels))
