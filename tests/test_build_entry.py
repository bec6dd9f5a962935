"""``__graft_entry__.build()`` in a tree that has no native files yet: one call, one process."""
import os
import shutil
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_build_in_a_clean_tree(tmp_path):
    tree = tmp_path / "tree"
    shutil.copytree(os.path.join(ROOT, "onnxruntime_b200"), tree / "onnxruntime_b200",
                    ignore=shutil.ignore_patterns("*.so", "build", "csrc", "__pycache__", "lib"))
    shutil.copy(os.path.join(ROOT, "__graft_entry__.py"), tree)
    # the compiler step puts the files of this tree in place
    script = f"""
import glob, os, shutil, sys
import __graft_entry__
from onnxruntime_b200 import build
def compiled(*args, **kwargs):
    os.makedirs('onnxruntime_b200/lib')
    for path in glob.glob({os.path.join(ROOT, "onnxruntime_b200")!r} + '/**/*.so', recursive=True):
        shutil.copy(path, os.path.join('onnxruntime_b200', os.path.relpath(path, {os.path.join(ROOT, "onnxruntime_b200")!r})))
build.build = compiled
import onnxruntime_b200
try:
    onnxruntime_b200.InferenceSession
    sys.exit('the copied tree is built already')
except ImportError:
    pass
__graft_entry__.build()
assert onnxruntime_b200.__file__.startswith(os.getcwd())
assert onnxruntime_b200.InferenceSession and 'CPUExecutionProvider' in onnxruntime_b200.get_available_providers()
try:
    onnxruntime_b200.no_such_name
    sys.exit('an unknown name was found')
except AttributeError:
    pass
"""
    env = {k: v for k, v in os.environ.items() if k != "PYTHONPATH"}
    done = subprocess.run([sys.executable, "-c", script], cwd=tree, env=env, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
