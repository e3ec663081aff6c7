"""bench.py as a source file: every function is defined once, and the headline
line's launch count is that of the kernels a run was seen to launch."""
import ast
import collections
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_functions_are_defined_once():
    with open(os.path.join(ROOT, "bench.py")) as fh:
        tree = ast.parse(fh.read())
    names = collections.Counter(node.name for node in tree.body if isinstance(node, (ast.FunctionDef, ast.ClassDef)))
    assert [name for name, count in names.items() if count > 1] == []


def test_launch_count(monkeypatch):
    import bench
    monkeypatch.delenv("KM_TC_CHUNKS", raising=False)
    # 169 kernels seen in a run of 5 iterations on 2,000,000 frames whose
    # iterations were launched one by one, without the loop's 4 steps
    assert bench.lloyd_launches(2_000_000, 5) == 169 + 4
    # two iterations keep no bounds: 29 kernels each, 4 before, a loop step
    assert bench.lloyd_launches(2_000_000, 2) == 2 * 29 + 4 + 1
