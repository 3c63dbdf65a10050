"""A test that calls the reference CPU kernel where it is not built is skipped;
other callers get an error."""
import unittest

import pytest

from conftest import load_golden
from oracle import oracle as O


@pytest.mark.parametrize("ns", [1, 60])
def test_the_absent_reference_skips(ns, monkeypatch):
    monkeypatch.setattr(O, "_ref_path", lambda ms64: None)
    P, prop, _ = load_golden("single_seed1")
    P.n_sources = ns
    with pytest.raises(RuntimeError) as e:
        O.ref_evaluate(P, prop)
    assert isinstance(e.value, unittest.SkipTest) and not O.ref_available(ns)
