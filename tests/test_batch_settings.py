"""The batch command says which of the asked-for launch settings are not in use."""
import pytest

from orkan_b200.batch import ignored_settings


@pytest.mark.parametrize("asked,note", [
    ({}, ""),
    ({"chunk": 12, "threads": 256, "ring": 2}, ""),
    ({"chunk": 12, "threads": 512, "ring": 1}, "not used: threads 512 (in use: 256), ring 1 (in use: 2)"),
    ({"chunk": 9}, "not used: chunk 9 (in use: 12)"),
])
def test_settings_not_in_use_are_named(asked, note):
    assert ignored_settings((12, 256, 2), **asked) == note
