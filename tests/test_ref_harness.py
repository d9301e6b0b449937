"""Which directories oracle/ref_harness.py takes for a checkout: none and an empty one
are absent, one with sources missing fails and names them."""
import os

import pytest

from oracle import ref_harness


def test_no_checkout_or_an_empty_one(tmp_path, monkeypatch):
    monkeypatch.delenv("VKZG_REFERENCE_DIR", raising=False)
    assert ref_harness.build() is None
    assert ref_harness.build(str(tmp_path / "nowhere")) is None
    assert ref_harness.build(str(tmp_path)) is None


def test_partial_checkout_fails(tmp_path):
    os.makedirs(tmp_path / "tests")
    (tmp_path / "tests" / "test.cpp").write_text("int main() { return 0; }\n")
    with pytest.raises(FileNotFoundError, match="tests/vectors.cpp.*bench/bench.cpp"):
        ref_harness.build(str(tmp_path))
