"""The tests that conftest skips in a build without the stream coders exist,
and they are skipped in such a build only."""
import importlib
import os

import pytest

from tests import conftest


@pytest.mark.parametrize("name", sorted(conftest.NEEDS_CODERS))
def test_listed_tests_exist(name):
    mod = importlib.import_module("tests." + name[:-3])
    assert all(callable(getattr(mod, t)) for t in conftest.NEEDS_CODERS[name])


def test_a_build_with_the_coders_skips_nothing():
    with_coders = os.path.exists(os.path.join(conftest.ROOT, "curc_b200", "_build", "libcurc_coders.a"))
    assert conftest.built_without_coders() == (not with_coders)
