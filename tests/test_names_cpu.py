"""Every test runs: a second function of one name in a module would replace the first before it is collected."""
import ast
from collections import Counter
from pathlib import Path

import pytest


@pytest.mark.parametrize("path", sorted(Path(__file__).resolve().parent.glob("test_*.py")), ids=lambda p: p.stem)
def test_names_are_unique(path):
    names = Counter(n.name for n in ast.parse(path.read_text()).body if isinstance(n, (ast.FunctionDef, ast.ClassDef)))
    assert not [n for n, k in names.items() if k > 1]
