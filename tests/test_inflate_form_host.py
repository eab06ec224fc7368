"""The inflate form that the library takes by itself (no kernel runs)."""

import pytest

from cubam_b200 import _lib, bgzf

L = _lib.lib


@pytest.fixture(autouse=True)
def restore_params():
    yield
    for key in (_lib.PARAM_SPLIT_MIN_JOBS, _lib.PARAM_INFLATE_FORM):
        L.cb_set_param(key, -1)


def test_no_least_number_of_jobs_until_one_is_set():
    assert [bgzf.inflate_form(0, n) for n in (0, 1, 8191, 8192, 1 << 40)] == [3] * 5


def test_small_members_take_form_1():
    """A rule on the mean size, and the workspace of the form that it names."""
    for n, small in ((1, 600), (39, 600), (8192, 600), (1 << 20, 600)):
        assert bgzf.inflate_form(0, n, n * small) == 1 and bgzf.inflate_form(0, n, n * (small + 1)) == 3
        assert bgzf.inflate_workspace_bytes(n, n * small) == int(L.cb_inflate_workspace_bytes())
        assert bgzf.inflate_workspace_bytes(n, n * (small + 1)) >= int(L.cb_inflate_split_workspace_bytes(n, n * (small + 1)))
        assert bgzf.inflate_form(3, n, n) == 3
        assert L.cb_set_param(_lib.PARAM_SPLIT_MIN_JOBS, _lib.SPLIT_MIN_JOBS_ANY) == _lib.OK
        assert bgzf.inflate_form(0, n, n * small) == 3
        L.cb_set_param(_lib.PARAM_SPLIT_MIN_JOBS, -1)


@pytest.mark.parametrize("least", [1, 100, 8191, 8192, 8193, 1 << 40])
def test_every_least_number_of_jobs_is_kept_to(least):
    assert L.cb_set_param(_lib.PARAM_SPLIT_MIN_JOBS, least) == _lib.OK
    assert L.cb_get_param(_lib.PARAM_SPLIT_MIN_JOBS) == least
    assert bgzf.inflate_form(0, least - 1) == 1 and bgzf.inflate_form(0, least) == 3 and bgzf.inflate_form(0) == 3
    assert bgzf.inflate_form(3, least - 1) == 3
    L.cb_set_param(_lib.PARAM_INFLATE_FORM, 2)
    assert bgzf.inflate_form(0, least - 1) == 2
    L.cb_set_param(_lib.PARAM_INFLATE_FORM, -1)
    for none in (_lib.SPLIT_MIN_JOBS_ANY, -1):
        assert L.cb_set_param(_lib.PARAM_SPLIT_MIN_JOBS, none) == _lib.OK
        assert bgzf.inflate_form(0, least - 1) == 3
