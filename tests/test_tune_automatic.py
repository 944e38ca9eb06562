"""The autotuner times the library's own schedule beside the explicit ones,
keeps it where it is at least as fast, and does not take measurements of
earlier schedules from its cache."""
import pytest

from gpu_deconvolution_b200 import autotune


@pytest.mark.parametrize("plane", [(128, 128), (512, 512), (1024, 1536), (1536, 1536), (4096, 4096)])
def test_automatic_schedule_is_a_candidate(plane):
    c = autotune.candidates(*plane)
    radix = (1, 2) if max(plane) > 1024 else (1,)
    assert all((0, 0, r) in c for r in radix)
    assert {k[0] for k in c} == {0, *autotune.pair_candidates(*plane)}
    assert len(set(c)) == len(c)


@pytest.mark.parametrize("auto_ms,automatic", [(0.9, True), (1.0, True), (1.1, False)])
def test_choice(auto_ms, automatic):
    e = autotune.choose({(0, 0, 1): auto_ms, (0, 0, 2): 3.0, (4, 8, 1): 1.0, (2, 8, 2): 1.2})
    assert e["automatic"] is automatic and (e["pairs_per_batch"], e["col_warps"]) == (4, 8)
    assert autotune.plan_settings(e) == ({"pairs_per_batch": 0, "col_warps": 0, "radix_step": 1} if automatic else
                                         {"pairs_per_batch": 4, "col_warps": 8, "radix_step": 1})


def test_entries_of_earlier_schedules_are_not_used(tmp_path):
    path = str(tmp_path / "tune.json")
    autotune.save_entry("B200|512x512|V4|u16", {"pairs_per_batch": 6, "col_warps": 8, "radix_step": 1}, path)
    assert autotune.cache_key("B200", 512, 512, 4, 16) not in autotune.load_cache(path)
