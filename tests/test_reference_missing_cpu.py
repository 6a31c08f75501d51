"""CPU: without the reference's solvers the oracle says so by an error of its own, for which tests
are skipped; with its sources at hand a missing library is a failure."""
import pytest

import oracle


def test_missing_reference(monkeypatch, tmp_path):
    monkeypatch.setattr(oracle, "_REF", str(tmp_path))
    monkeypatch.setattr(oracle, "_ref_eik", None)
    monkeypatch.setattr(oracle, "reference_src", lambda: None)
    with pytest.raises(oracle.ReferenceNotBuilt):
        oracle.ref_catch_parameter("key", "file")
    monkeypatch.setattr(oracle, "reference_src", lambda: str(tmp_path))
    with pytest.raises(OSError) as e:
        oracle.ref_catch_parameter("key", "file")
    assert not isinstance(e.value, oracle.ReferenceNotBuilt)
