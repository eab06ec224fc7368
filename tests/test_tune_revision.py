"""Tuned values are used by the kernels they were tuned for (no kernel runs)."""

from cubam_b200 import tune


def test_an_entry_tuned_for_other_kernels_is_not_applied(tmp_path):
    path = tmp_path / "tune.json"
    before = tune.current()
    key = tune.shape_key(1024, 1 << 26)
    old = {"params": dict(before, inflate_form=1, copy_warps=24)}
    assert f"|rev{tune.REVISION}" in key
    tune.save_cache({key.replace(f"|rev{tune.REVISION}", ""): old, key.replace(f"|rev{tune.REVISION}", "|rev1"): old}, path)
    assert tune.apply_cached(1024, 1 << 26, path) is None and tune.current() == before
    tune.save_cache({**tune.load_cache(path), key: {"params": before}}, path)
    assert tune.apply_cached(1024, 1 << 26, path) == before
