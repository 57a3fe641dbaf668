"""CPU: the library and the model drivers need neither torch nor the native host module; the ops take that module when it is there."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NO_TORCH = "import sys; sys.modules['torch'] = None\n"


def _run(code, root=ROOT, **env):
    r = subprocess.run([sys.executable, "-W", "ignore", "-c", code], cwd=root, env=dict(os.environ, PYTHONPATH=root, **env), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout.split()


def test_library_without_torch(lib):
    out = _run(NO_TORCH + "from zhilight_b200.llama import LlamaDecoder\nfrom zhilight_b200 import engine, registry, dist, _lib\n"
               "print(_lib.load().zl_version() >= 100, _lib.host, 'torch._C' in sys.modules)")
    assert out == ["True", "None", "False"]


@pytest.mark.parametrize("first", ["from zhilight_b200 import ops", "pass"])
def test_module_comes_with_the_ops(lib, first):
    """Whichever of the library and ops.py comes first."""
    assert _run(first + "\nfrom zhilight_b200 import _lib\n_lib.load()\nfrom zhilight_b200 import ops\nprint(_lib.host is not None)") == ["True"]


def test_building_does_not_import_torch(lib):
    """With everything built: it costs a program seconds."""
    assert _run("import sys\nfrom zhilight_b200 import build\nbuild.build()\nprint('torch' in sys.modules)") == ["False"]


@pytest.fixture
def bare(tmp_path, lib):
    """A checkout that has the CUDA library and nothing else built."""
    root = tmp_path / "bare"
    shutil.copytree(os.path.join(ROOT, "zhilight_b200"), root / "zhilight_b200",
                    ignore=shutil.ignore_patterns("build", "__pycache__", "_host*", "libzhilight_b200.so"))
    shutil.copytree(os.path.join(ROOT, "include"), root / "include")
    os.symlink(os.path.join(ROOT, "zhilight_b200", "libzhilight_b200.so"), root / "zhilight_b200" / "libzhilight_b200.so")
    return str(root)


def test_ops_without_the_module(bare):
    assert _run("from zhilight_b200 import ops, _lib\nprint(_lib.load().zl_version() >= 100, _lib.host)", bare) == ["True", "None"]


def test_build_without_torch_or_compiler(bare):
    code = "from zhilight_b200 import build\nprint(build.build_host(), build.build() == build.LIB_PATH)"
    assert _run("import importlib.util as u\nf = u.find_spec\nu.find_spec = lambda n, *a: None if n == 'torch' else f(n, *a)\n" + code, bare) == ["None", "True"]
    assert _run(code, bare, PATH="/nonexistent") == ["None", "True"]
