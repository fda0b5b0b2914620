"""bench.py names the kernel that a tile shape stands for: its labels against the
table of FP32 shapes in mo-dmft_gb300/csrc/hv.cu, and no definition of the
file overwritten by a second one."""
import ast
import importlib.util
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_labels():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    with open(os.path.join(ROOT, "mo-dmft_gb300", "csrc", "hv.cu")) as f:
        table = re.search(r"kVarF32\[\] = \{(.*?)\};", f.read(), re.S).group(1)
    shapes = re.findall(r"\{(\d+), (\d+), (\d+), (\d+)(, true)?\}", table)
    assert len(shapes) >= 10
    for *shape, wide in shapes:
        shape = tuple(int(v) for v in shape)
        name = bench.kernel_name(shape)
        assert ("k_hv_wide" in name) == bool(wide), (shape, name)
        assert ("k_hv_row" == name) == (shape[0] == 1 and shape[3] == 0)
        assert ("k_hv_down_rows" in name) == (shape[3] == 4)


def test_defined_once():
    with open(os.path.join(ROOT, "bench.py")) as f:
        body = ast.parse(f.read()).body
    names = [n.name for n in body if isinstance(n, (ast.FunctionDef, ast.ClassDef))]
    names += [t.id for n in body if isinstance(n, ast.Assign) for t in n.targets if isinstance(t, ast.Name)]
    assert sorted(names) == sorted(set(names))
