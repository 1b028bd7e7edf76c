"""A test that builds the reference without asking whether it is there is skipped, not failed."""
import unittest

import pytest

from oracle import pyoracle as po
from physik_b200 import meshes


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_a_missing_build_skips(precision, monkeypatch, tmp_path):
    monkeypatch.setattr(po, "HERE", str(tmp_path))
    with pytest.raises(unittest.SkipTest):
        po.Reference(meshes.small_box(1, 1, 1), precision)
    with pytest.raises(unittest.SkipTest):
        po._ref_lib(precision)

