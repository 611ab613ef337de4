"""Tests that compare with the reference are skipped for one reason only: its sources were absent at the build."""
import importlib.util
import os

import pytest

import oracle
from conftest import ROOT


def test_reference_oracle_is_built_where_its_sources_are():
    assert oracle.ref_available() or not oracle.ref_expected()


@pytest.mark.parametrize("record,expected", [("present\n", True), ("absent\n", False)])
def test_missing_oracle_is_absent_or_an_error(monkeypatch, tmp_path, record, expected):
    path = tmp_path / "reference_sources"
    path.write_text(record)
    monkeypatch.setattr(oracle, "RECORD", str(path))
    monkeypatch.setattr(oracle, "REF_LIB", str(tmp_path / "libccref.so"))
    monkeypatch.setattr(oracle, "_REF", None)
    assert oracle.ref_expected() == expected
    with pytest.raises(OSError if expected else oracle.ReferenceAbsent):
        oracle.ref_lib()


def test_named_tree_without_sources_fails_the_build(monkeypatch, tmp_path):
    spec = importlib.util.spec_from_file_location("graft_entry", os.path.join(ROOT, "__graft_entry__.py"))
    entry = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(entry)
    monkeypatch.setenv("CC_REFERENCE_TREE", str(tmp_path))
    with pytest.raises(RuntimeError, match="no reference sources"):
        entry.reference_tree()
    (tmp_path / "potential").mkdir()
    assert entry.reference_tree() == str(tmp_path)
